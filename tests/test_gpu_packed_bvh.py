"""The packed BVH of the wavefront kernels and the engine against the plain kernel, which reads the uploaded nodes:
trees at the limits of the packed form (largest leaf, boxes that are not their children's union, inverted boxes,
unreachable nodes) and rays along an axis.  The accumulations must be equal bit for bit."""
import ctypes as C

import numpy as np
import pytest

import pathtracer as pt
from pathtracer import abi
from pathtracer.engine import Engine

pytestmark = pytest.mark.gpu

NODE = np.dtype([("min", "<f4", 3), ("first", "<u4"), ("max", "<f4", 3), ("count", "<u4")])


def merged(nodes, most):
    """The tree with every subtree of at most `most` triangles as one leaf, every node reachable, child pairs in order."""
    size, start = {}, {}

    def measure(i):
        n = nodes[i]
        if n["count"]:
            size[i], start[i] = int(n["count"]), int(n["first"])
        else:
            left = int(n["first"])
            measure(left)
            measure(left + 1)
            size[i], start[i] = size[left] + size[left + 1], min(start[left], start[left + 1])

    measure(0)
    out, todo = [nodes[0].copy()], [(0, 0)]
    while todo:
        new, old = todo.pop()
        if size[old] <= most or nodes[old]["count"]:
            out[new]["first"], out[new]["count"] = start[old], size[old]
            continue
        left = int(nodes[old]["first"])
        out[new]["first"], out[new]["count"] = len(out), 0
        todo += [(len(out) + 1, left + 1), (len(out), left)]
        out += [nodes[left].copy(), nodes[left + 1].copy()]
    return np.array(out, NODE)


def loosened(nodes):
    """Every seventh box larger than its triangles need, so that it is not the union of its children's."""
    out = nodes.copy()
    out["max"][3::7] += np.float32(0.25)
    out["min"][5::7] -= np.float32(0.125)
    return out


def inverted(nodes):
    """Every eleventh box with its x planes exchanged."""
    out = nodes.copy()
    out["min"][4::11, 0], out["max"][4::11, 0] = nodes["max"][4::11, 0], nodes["min"][4::11, 0]
    return out


def with_unreachable(nodes):
    """Two more nodes that nothing refers to, one of them an interior node over the root's children."""
    extra = nodes[:2].copy()
    extra[1]["first"] = 0xfffffff0
    return np.concatenate([nodes, extra])


FORMS = {"as built": lambda n: n, "leaves of 14": lambda n: merged(n, 14), "leaves of 15": lambda n: merged(n, 15),
         "one leaf": lambda n: merged(n, 1 << 30), "loose boxes": loosened, "inverted boxes": inverted,
         "unreachable nodes": with_unreachable}


@pytest.fixture(scope="module")
def worlds():
    # (the 36-triangle room is small enough to be one leaf)
    out = {"room": pt.World.cornell_box(),
           "field": pt.World.procedural(seed=3, grid_x=24, grid_z=16, boxes=40, spheres=2, sphere_subdivision=2,
                                        emissive_triangles=8, skybox_width=32, skybox_height=16)}
    return {name: (w, w.take_updates()) for name, w in out.items()}


def updates_with(worlds, name, form, camera=None):
    full = worlds[name][1]
    scene = abi.SceneUpload.from_buffer_copy(full.scene.contents)
    raw = C.string_at(scene.bvh_nodes, 32 * scene.node_count)
    nodes = np.ascontiguousarray(FORMS[form](np.frombuffer(raw, NODE).copy()))
    scene.bvh_nodes = C.cast(nodes.ctypes.data, C.POINTER(abi.BvhNode))
    scene.node_count = len(nodes)
    u = abi.WorldUpdates.from_buffer_copy(full)
    u.scene = C.pointer(scene)
    if camera is not None:
        u.camera = C.pointer(camera)
    return u, (scene, nodes, camera)


def accumulations(u, size, spp, bounces):
    out = []
    for kernel in (abi.PT_KERNEL_PLAIN, abi.PT_KERNEL_WAVEFRONT):
        t = pt.PathTracer(u, size)
        t.set_kernel(kernel)
        t.set_max_bounces(bounces)
        assert t.trace(spp) == spp
        out.append(t.read_tile(abi.PT_TILE_ACCUMULATION))
        t.close()
    return out


@pytest.mark.parametrize("form", [f for f in FORMS if f != "one leaf"])
def test_tree_forms_equal_plain(worlds, form):
    u, _keep = updates_with(worlds, "field", form)
    plain, wave = accumulations(u, (96, 64), 4, 6)
    assert plain[..., :3].max() > 0
    assert plain.tobytes() == wave.tobytes()


@pytest.mark.parametrize("form", ["as built", "one leaf"])
def test_small_trees_equal_plain(worlds, form):
    u, _keep = updates_with(worlds, "room", form)
    plain, wave = accumulations(u, (64, 64), 4, 6)
    assert plain.tobytes() == wave.tobytes()


@pytest.mark.parametrize("form", ["as built", "loose boxes"])
@pytest.mark.parametrize("flat", ["horizontal", "both"])
def test_axis_parallel_rays_equal_plain(worlds, form, flat):
    """Cameras without a horizontal (and vertical) extent: every camera ray has one (two) zero components."""
    full = worlds["field"][1]
    cam = abi.Camera.from_buffer_copy(full.camera.contents)
    cam.horizontal[:] = [0.0] * 4
    cam.lower_left_corner_minus_position[:] = [0.0, -0.4, -1.0, 0.0]
    cam.vertical[:] = [0.0, 0.5, 0.0, 0.0]
    if flat == "both":
        cam.lower_left_corner_minus_position[:] = [0.0, -1.0, 0.0, 0.0]
        cam.vertical[:] = [0.0] * 4
    u, _keep = updates_with(worlds, "field", form, cam)
    plain, wave = accumulations(u, (33, 20), 2, 4)
    assert plain.tobytes() == wave.tobytes()


def test_engine_mixes_packed_and_unpacked_scenes(worlds):
    """Scenes whose tree fits the packed form and scenes whose tree does not, in the same waves."""
    eng = Engine(wave_paths=1 << 14, tile_size=16)
    jobs, keep = [], []
    for form in ("as built", "leaves of 15", "loose boxes", "unreachable nodes"):
        u, k = updates_with(worlds, "field", form)
        keep.append(k)
        sid = eng.add_scene(u)
        cam = abi.Camera.from_buffer_copy(u.camera.contents)
        jobs.append((u, eng.submit(sid, cam, 48, 40, 3, 5)))
    eng.wait_idle(timeout_ms=60000)
    for u, job in jobs:
        plain, _ = accumulations(u, (48, 40), 3, 5)
        assert eng.read(job, 48, 40, abi.PT_TILE_ACCUMULATION).tobytes() == plain.tobytes()
    eng.close()
