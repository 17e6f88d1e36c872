"""The checks of a large scene upload on the GPU decide as the host's do: each malformed tree or material index is
refused with its code and message and leaves the world untouched, and the valid trees that the GPU's checks do not
know (children before their parent, nodes that nothing reaches) render the same bits."""
import ctypes as C

import numpy as np
import pytest

import pathtracer as pt
from pathtracer import abi

pytestmark = pytest.mark.gpu

NODE = np.dtype([("lo", "<f4", 3), ("left_first", "<u4"), ("hi", "<f4", 3), ("tri_count", "<u4")])


@pytest.fixture(scope="module")
def world():
    w = pt.World.procedural(seed=3, grid_x=128, grid_z=96, boxes=400, spheres=40, sphere_subdivision=3,
                            emissive_triangles=32, skybox_width=64, skybox_height=32)
    w.set_aspect_ratio(1.0)
    w.edit_camera(yaw=0.1, pitch=-0.35)
    updates = w.take_updates()
    s = updates.scene.contents
    assert s.node_count >= 1 << 15
    nodes = np.frombuffer(C.string_at(s.bvh_nodes, 32 * s.node_count), NODE)
    yield w, updates, nodes


def with_scene(updates, nodes=None, attributes=None):
    scene = abi.SceneUpload.from_buffer_copy(updates.scene.contents)
    if nodes is not None:
        scene.bvh_nodes = C.cast(nodes.ctypes.data, C.POINTER(abi.BvhNode))
        scene.node_count = len(nodes)
    if attributes is not None:
        scene.attributes = C.cast(attributes.ctypes.data, C.POINTER(abi.TriangleAttribute))
    u = abi.WorldUpdates.from_buffer_copy(updates)
    u.scene = C.pointer(scene)
    return u, (scene, nodes, attributes)


def render(tr):
    tr.set_tile((64, 64), (0, 0), (64, 64))
    tr.trace(2)
    return tr.read_tile(abi.PT_TILE_ACCUMULATION).view(np.uint32)


def chain(nodes, levels):
    """nodes with the first right-hand leaf replaced by a chain `levels` deep, appended at the end"""
    leaf = int(np.flatnonzero(nodes["tri_count"] > 0)[0])
    more = np.repeat(nodes[leaf:leaf + 1], 2 * levels)
    out = np.concatenate([nodes, more])
    out["left_first"][leaf], out["tri_count"][leaf] = len(nodes), 0
    for k in range(levels - 1):
        at = len(nodes) + 2 * k
        out["left_first"][at], out["tri_count"][at] = at + 2, 0
    return out


def depth_of(nodes, i):
    parent = {}
    for p in np.flatnonzero(nodes["tri_count"] == 0):
        l = int(nodes["left_first"][p])
        parent[l] = parent[l + 1] = int(p)
    d = 0
    while i:
        i, d = parent[i], d + 1
    return d


def bad_tree(kind, nodes, triangles):
    n = nodes.copy()
    inner = np.flatnonzero(n["tri_count"] == 0)
    leaves = np.flatnonzero(n["tri_count"] > 0)
    if kind == "twice":
        n["left_first"][inner[-1]] = n["left_first"][inner[1]]  # before its parent too: the general walk
    elif kind == "twice, in order":
        n["left_first"][inner[1]] = n["left_first"][inner[2]]
    elif kind == "child":
        n["left_first"][inner[-1]] = len(n) - 1
    elif kind == "leaf":
        n["left_first"][leaves[-1]] = triangles - int(n["tri_count"][leaves[-1]]) + 1
    elif kind == "deep":
        n = chain(n, 65 - depth_of(n, int(leaves[0])))
    return n


@pytest.mark.parametrize("kind,code,text", [
    ("twice", abi.PT_ERR_INVALID_ARG, "reached twice"), ("twice, in order", abi.PT_ERR_INVALID_ARG, "reached twice"),
    ("child", abi.PT_ERR_INVALID_ARG, "child index outside"), ("leaf", abi.PT_ERR_INVALID_ARG, "leaf triangle range"),
    ("deep", abi.PT_ERR_OUT_OF_LIMITS, "deeper than the 64-entry"),
    ("material", abi.PT_ERR_INVALID_ARG, "material index outside")])
def test_malformed_scene_refused(world, kind, code, text):
    _, updates, nodes = world
    s = updates.scene.contents
    tr = pt.PathTracer(updates, (64, 64))
    want = render(tr)
    if kind == "material":
        attributes = np.frombuffer(C.string_at(s.attributes, 112 * s.triangle_count), np.uint32).copy().reshape(-1, 28)
        attributes[-1, 0] = s.material_count
        bad, keep = with_scene(updates, attributes=attributes)
    else:
        bad, keep = with_scene(updates, bad_tree(kind, nodes, s.triangle_count))
    with pytest.raises(pt.PathTracerError) as e:
        tr.apply_updates(bad)
    assert e.value.code == code and text in e.value.message, (e.value.code, e.value.message)
    np.testing.assert_array_equal(render(tr), want)
    tr.close()


@pytest.mark.parametrize("kind", ["order", "unreached", "deepest"])
def test_valid_scene_renders_the_same(world, kind):
    _, updates, nodes = world
    tr = pt.PathTracer(updates, (64, 64))
    want = render(tr)
    n = nodes.copy()
    if kind == "order":  # the child pairs in another order
        pairs = (len(n) - 1) // 2
        place = np.random.default_rng(1).permutation(pairs)
        n[1:].reshape(-1, 2)[place] = nodes[1:].reshape(-1, 2)
        inner = n["tri_count"] == 0
        n["left_first"][inner] = 2 * place[(n["left_first"][inner] - 1) // 2] + 1
    elif kind == "unreached":
        n = np.concatenate([n, n[-2:]])
    else:  # as deep as the stack allows, the chain's leaves copies of one leaf (a later equal hit changes nothing)
        leaf = int(np.flatnonzero(n["tri_count"] > 0)[0])
        n = chain(n, 64 - depth_of(n, leaf))
    tr.apply_updates(with_scene(updates, n)[0])
    np.testing.assert_array_equal(render(tr), want)
    tr.close()
