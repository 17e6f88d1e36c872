"""Boxes that are not numbers, in part or wholly, and infinite ones, in a tree that is uploaded: every kernel visits the
nodes that the reference's slab test accepts (a box without any number is rejected, with what is below it).  Against
the plain kernel, which runs that test as written: images bit for bit, and the records of every visit."""
import ctypes as C

import numpy as np
import pytest

import pathtracer as pt
import test_gpu_packed_bvh as trees
from pathtracer import abi
from pathtracer.engine import Engine

pytestmark = pytest.mark.gpu

NAN, INF = np.float32("nan"), np.float32("inf")


def boxless(nodes):
    nodes["min"][3::9] = nodes["max"][3::9] = NAN
    return nodes


def half_boxless(nodes):
    """One side of some boxes, one axis of others."""
    nodes["max"][3::9] = NAN
    nodes["min"][4::9, 1] = nodes["max"][4::9, 1] = NAN
    return nodes


def endless(nodes):
    nodes["min"][3::9], nodes["max"][3::9] = -INF, INF
    nodes["max"][4::9, 2] = INF
    return nodes


FORMS = {"no box": boxless, "no box, leaves of 15": lambda n: boxless(trees.merged(n, 15)), "half a box": half_boxless,
         "infinite": endless, "infinite, leaves of 15": lambda n: endless(trees.merged(n, 15))}


@pytest.fixture(scope="module")
def world():
    w = pt.World.procedural(seed=3, grid_x=24, grid_z=16, boxes=40, spheres=2, sphere_subdivision=2,
                            emissive_triangles=8, skybox_width=32, skybox_height=16)
    return w, w.take_updates()


def updates_with(world, form):
    scene = abi.SceneUpload.from_buffer_copy(world[1].scene.contents)
    raw = C.string_at(scene.bvh_nodes, 32 * scene.node_count)
    nodes = np.ascontiguousarray(FORMS[form](np.frombuffer(raw, trees.NODE).copy()))
    scene.bvh_nodes = C.cast(nodes.ctypes.data, C.POINTER(abi.BvhNode))
    scene.node_count = len(nodes)
    u = abi.WorldUpdates.from_buffer_copy(world[1])
    u.scene = C.pointer(scene)
    return u, (scene, nodes)


@pytest.mark.parametrize("form", FORMS)
def test_images_equal_plain(world, form):
    u, _keep = updates_with(world, form)
    plain, wave = trees.accumulations(u, (96, 64), 4, 6)
    assert plain[..., :3].max() > 0
    assert plain.tobytes() == wave.tobytes()


@pytest.mark.parametrize("form", FORMS)
def test_records_equal_plain(world, form):
    u, _keep = updates_with(world, form)
    records = []
    for kernel in (abi.PT_KERNEL_PLAIN, abi.PT_KERNEL_WAVEFRONT):
        t = pt.PathTracer(u, (40, 30))
        t.set_kernel(kernel)
        t.set_max_bounces(4)
        records.append(t.trace_recorded(2).tobytes())
        t.close()
    assert records[0] == records[1]


def test_engine_equals_plain(world):
    eng = Engine(wave_paths=1 << 14, tile_size=16)
    jobs, keep = [], []
    for form in FORMS:
        u, k = updates_with(world, form)
        keep.append(k)
        jobs.append((u, eng.submit(eng.add_scene(u), abi.Camera.from_buffer_copy(u.camera.contents), 48, 40, 3, 5)))
    eng.wait_idle(timeout_ms=60000)
    for u, job in jobs:
        plain, _ = trees.accumulations(u, (48, 40), 3, 5)
        assert eng.read(job, 48, 40, abi.PT_TILE_ACCUMULATION).tobytes() == plain.tobytes()
    eng.close()
