"""Trees in which some boxes are not the union of their children's, so that a packed BVH holds no planes of those nodes:
few of them (the packed traversal visits them from the uploaded nodes), as many as the packed form is taken with (one
in 128 nodes), one more, and most.  Against the plain kernel, bit for bit, as tiles, along an axis and in engine waves."""
import ctypes as C

import numpy as np
import pytest

import pathtracer as pt
import test_gpu_packed_bvh as trees
from pathtracer import abi
from pathtracer.engine import Engine

pytestmark = pytest.mark.gpu


def union_of_children(nodes):
    inner = np.flatnonzero(nodes["count"] == 0)
    left = nodes["first"][inner].astype(np.int64)
    lo, hi = np.minimum(nodes["min"][left], nodes["min"][left + 1]), np.maximum(nodes["max"][left], nodes["max"][left + 1])
    return inner, (lo == nodes["min"][inner]).all(1) & (hi == nodes["max"][inner]).all(1)


def leaves_of(nodes):
    """One leaf for each interior node over two leaves."""
    inner = np.flatnonzero(nodes["count"] == 0)
    left = nodes["first"][inner].astype(np.int64)
    pairs = inner[(nodes["count"][left] > 0) & (nodes["count"][left + 1] > 0)]
    return nodes["first"][pairs].astype(np.int64)


def changed(nodes, count, how):
    """`count` leaves changed, each below an interior node of its own, which is then no union any more."""
    out = nodes.copy()
    at = leaves_of(nodes)
    at = at[:: max(1, len(at) // count)][:count]
    assert len(at) == count
    if how == "loose":
        out["max"][at] += np.float32(8.0)
    elif how == "inverted":
        # (the axis of the largest extent: a flat box is its own inverse)
        axis = (nodes["max"][at] - nodes["min"][at]).argmax(1)
        out["min"][at, axis], out["max"][at, axis] = nodes["max"][at, axis], nodes["min"][at, axis]
    else:
        out["min"][at] = out["max"][at] = np.float32("nan")
    inner, exact = union_of_children(out)
    if how == "loose":
        assert int((~exact).sum()) == count
    return out


COUNTS = {"three": lambda n: 3, "at the line": lambda n: n // 128, "beyond it": lambda n: n // 128 + 1, "most": lambda n: n // 8}
FORMS = {(how, many): (lambda n, how=how, f=f: changed(n, f(len(n)), how))
         for how in ("loose", "inverted", "no box") for many, f in COUNTS.items()}


@pytest.fixture(scope="module")
def world():
    w = pt.World.procedural(seed=3, grid_x=24, grid_z=16, boxes=40, spheres=2, sphere_subdivision=2,
                            emissive_triangles=8, skybox_width=32, skybox_height=16)
    updates = w.take_updates()
    nodes = np.frombuffer(C.string_at(updates.scene.contents.bvh_nodes, 32 * updates.scene.contents.node_count), trees.NODE)
    assert union_of_children(nodes)[1].all()  # the builder's own boxes are unions
    return w, updates


def updates_with(world, form, camera=None):
    scene = abi.SceneUpload.from_buffer_copy(world[1].scene.contents)
    raw = C.string_at(scene.bvh_nodes, 32 * scene.node_count)
    nodes = np.ascontiguousarray(FORMS[form](np.frombuffer(raw, trees.NODE).copy()))
    scene.bvh_nodes = C.cast(nodes.ctypes.data, C.POINTER(abi.BvhNode))
    u = abi.WorldUpdates.from_buffer_copy(world[1])
    u.scene = C.pointer(scene)
    if camera is not None:
        u.camera = C.pointer(camera)
    return u, (scene, nodes, camera)


@pytest.mark.parametrize("form", FORMS, ids=" ".join)
def test_tiles_equal_plain(world, form):
    u, _keep = updates_with(world, form)
    plain, wave = trees.accumulations(u, (96, 64), 4, 6)
    assert plain[..., :3].max() > 0
    assert plain.tobytes() == wave.tobytes()


@pytest.mark.parametrize("form", [f for f in FORMS if f[1] == "at the line"], ids=" ".join)
def test_axis_parallel_rays_equal_plain(world, form):
    cam = abi.Camera.from_buffer_copy(world[1].camera.contents)
    cam.horizontal[:] = [0.0] * 4
    cam.lower_left_corner_minus_position[:] = [0.0, -0.4, -1.0, 0.0]
    cam.vertical[:] = [0.0, 0.5, 0.0, 0.0]
    u, _keep = updates_with(world, form, cam)
    plain, wave = trees.accumulations(u, (33, 20), 2, 4)
    assert plain.tobytes() == wave.tobytes()


def test_uploads_in_a_row(world):
    """The form is chosen anew for each upload."""
    t = pt.PathTracer(world[1], (64, 48))
    t.set_max_bounces(5)
    for form in (("loose", "most"), ("loose", "three"), ("no box", "beyond it"), ("inverted", "at the line")):
        u, _keep = updates_with(world, form)
        images = []
        for kernel in (abi.PT_KERNEL_PLAIN, abi.PT_KERNEL_WAVEFRONT):
            t.set_kernel(kernel)
            t.apply_updates(u)
            t.set_tile((64, 48), (0, 0), (64, 48))
            assert t.trace(3) == 3
            images.append(t.read_tile(abi.PT_TILE_ACCUMULATION).tobytes())
        assert images[0] == images[1]
    t.close()


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
