"""Small groups of paths, whose later rounds one kernel finishes, against the plain kernel: group sizes on both sides of
the lines at which that kernel takes over (from the first round, from the second, from a round of few hits, from the
sixth, never), with no bounce, one, and more than a record holds, in a closed room (every path lives on), an open field
(paths leave), a scene whose rays draw random numbers, and on the 8-wide BVH.  Equal bit for bit."""
import numpy as np
import pytest

import pathtracer as pt
from pathtracer import abi
from pathtracer.engine import Engine
from worlds import non_opaque_world

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def worlds():
    out = {"room": pt.World.cornell_box(),
           "field": pt.World.procedural(seed=3, grid_x=24, grid_z=16, boxes=40, spheres=2, sphere_subdivision=2,
                                        emissive_triangles=8, skybox_width=32, skybox_height=16),
           "coverage": non_opaque_world()}
    return {name: (w, w.take_updates()) for name, w in out.items()}


def accumulation(u, size, spp, bounces, kernel, precision=0, calls=1):
    t = pt.PathTracer(u, size)
    t.set_kernel(kernel)
    if precision:
        t.set_precision(precision)
    t.set_max_bounces(bounces)
    for _ in range(calls):
        assert t.trace(spp) == spp
    out = t.read_tile(abi.PT_TILE_ACCUMULATION)
    t.close()
    return out


@pytest.mark.parametrize("bounces", [0, 1, 5, 16])
@pytest.mark.parametrize("scene,size,spp", [
    ("field", (1, 1), 1), ("field", (31, 7), 3), ("room", (160, 120), 1), ("coverage", (97, 61), 5),
    ("room", (128, 64), 16), ("field", (129, 64), 16),      # 2^17 paths, and a few more
    ("field", (128, 128), 16), ("room", (129, 128), 16),    # 2^18
    ("coverage", (300, 217), 8), ("field", (512, 256), 16),  # 2^21
    ("field", (513, 256), 16)])
def test_equal_to_the_plain_kernel(worlds, scene, size, spp, bounces):
    u = worlds[scene][1]
    plain = accumulation(u, size, spp, bounces, abi.PT_KERNEL_PLAIN)
    wave = accumulation(u, size, spp, bounces, abi.PT_KERNEL_WAVEFRONT)
    assert bounces == 0 or size == (1, 1) or plain[..., :3].max() > 0
    assert plain.tobytes() == wave.tobytes()


@pytest.mark.parametrize("size,spp", [((33, 21), 2), ((128, 127), 16), ((300, 217), 8)])
def test_wide_form(worlds, size, spp):
    u = worlds["field"][1]
    plain = accumulation(u, size, spp, 8, abi.PT_KERNEL_PLAIN)
    wave = accumulation(u, size, spp, 8, abi.PT_KERNEL_WAVEFRONT, abi.PT_PRECISION_WIDE_BVH)
    assert plain.tobytes() == wave.tobytes()


@pytest.mark.parametrize("size", [(64, 64), (65, 64)])
def test_groups_beside_one_another(worlds, size):
    """Consecutive calls, whose groups overlap, on both sides of 2^16 paths a group."""
    u = worlds["room"][1]
    plain = accumulation(u, size, 16, 8, abi.PT_KERNEL_PLAIN, calls=5)
    wave = accumulation(u, size, 16, 8, abi.PT_KERNEL_WAVEFRONT, calls=5)
    assert plain.tobytes() == wave.tobytes()


@pytest.mark.parametrize("size,spp", [((40, 30), 1), ((129, 127), 10), ((300, 217), 8), ((520, 258), 16)])
@pytest.mark.parametrize("scene", ["room", "field", "coverage"])
def test_waves_of_every_size(worlds, scene, size, spp):
    """One request per wave: up to 2^17, 2^18 and 2^21 paths, and more."""
    u = worlds[scene][1]
    eng = Engine(wave_paths=1 << 22)
    cam = abi.Camera.from_buffer_copy(u.camera.contents)
    job = eng.submit(eng.add_scene(u), cam, *size, spp, 7)
    eng.wait_idle(timeout_ms=60000)
    plain = accumulation(u, size, spp, 7, abi.PT_KERNEL_PLAIN)
    assert eng.read(job, *size, abi.PT_TILE_ACCUMULATION).tobytes() == plain.tobytes()
    eng.close()


def test_waves_of_jobs_of_different_depths(worlds):
    """Small jobs of all three scenes and depths 0..9 in the same waves."""
    eng = Engine(wave_paths=1 << 20, tile_size=16)
    ids = {name: eng.add_scene(u) for name, (_, u) in worlds.items()}
    jobs = []
    for depth in range(10):
        name = sorted(worlds)[depth % 3]
        u = worlds[name][1]
        cam = abi.Camera.from_buffer_copy(u.camera.contents)
        jobs.append((u, depth, eng.submit(ids[name], cam, 30 + depth, 23, 3, depth)))
    eng.wait_idle(timeout_ms=60000)
    for u, depth, job in jobs:
        plain = accumulation(u, (30 + depth, 23), 3, depth, abi.PT_KERNEL_PLAIN)
        assert eng.read(job, 30 + depth, 23, abi.PT_TILE_ACCUMULATION).tobytes() == plain.tobytes()
    eng.close()
