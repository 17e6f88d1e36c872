"""Scenes of few nodes and many triangles, whose uploads the host checks: the tree and the skybox aliases beside the
material indices, which several threads scan from 2^18 triangles on.  What is wrong anywhere is refused with its
message and leaves the world untouched, and the first of several faults is the one named."""
import ctypes as C

import numpy as np
import pytest

import pathtracer as pt
from pathtracer import abi

pytestmark = pytest.mark.gpu

NODE = np.dtype([("lo", "<f4", 3), ("left_first", "<u4"), ("hi", "<f4", 3), ("tri_count", "<u4")])


def upload(base, triangles, nodes, material_at=None, alias=None):
    """`triangles` copies of the base scene's first triangle, in `nodes` leaves below a balanced tree."""
    s = abi.SceneUpload.from_buffer_copy(base.scene.contents)
    geometry = np.tile(np.frombuffer(C.string_at(s.geometries, 36), np.uint32), (triangles, 1))
    attributes = np.tile(np.frombuffer(C.string_at(s.attributes, 112), np.uint32), (triangles, 1))
    if material_at is not None:
        attributes[material_at, 0] = s.material_count
    tree = np.zeros(2 * nodes - 1, NODE)
    tree["lo"], tree["hi"] = -9.0, 9.0
    inner = np.arange(nodes - 1)
    tree["left_first"][inner] = 2 * inner + 1
    bounds = triangles * np.arange(nodes + 1) // nodes
    tree["left_first"][nodes - 1:], tree["tri_count"][nodes - 1:] = bounds[:-1], np.diff(bounds)
    s.geometries = C.cast(geometry.ctypes.data, type(s.geometries))
    s.attributes = C.cast(attributes.ctypes.data, type(s.attributes))
    s.bvh_nodes = C.cast(tree.ctypes.data, C.POINTER(abi.BvhNode))
    s.triangle_count, s.node_count = triangles, len(tree)
    u = abi.WorldUpdates.from_buffer_copy(base)
    u.scene = C.pointer(s)
    keep = [s, geometry, attributes, tree]
    if alias is not None:
        sky = type(base.skybox.contents).from_buffer_copy(base.skybox.contents)
        table = np.frombuffer(C.string_at(sky.alias_table, 12 * sky.alias_count), np.uint32).copy().reshape(-1, 3)
        field = [f for f, _ in abi.SkyboxAliasEntry._fields_].index("alias_index")
        table[-1, field] = alias
        sky.alias_table = C.cast(table.ctypes.data, type(sky.alias_table))
        u.skybox = C.pointer(sky)
        keep += [sky, table]
    return u, keep, tree


@pytest.fixture(scope="module")
def world():
    w = pt.World.procedural(seed=3, grid_x=24, grid_z=16, boxes=40, spheres=2, sphere_subdivision=2,
                            emissive_triangles=8, skybox_width=256, skybox_height=128)
    return w, w.take_updates()


@pytest.mark.parametrize("triangles,nodes", [(5000, 1), (16383, 9000), (16384, 9000), ((1 << 18) - 1, 16), (1 << 18, 16),
                                             ((1 << 18) + 5, 9000)])
def test_faults_are_refused(world, triangles, nodes):
    base = world[1]
    tr = pt.PathTracer(base, (32, 32))
    tr.trace(1)
    want = tr.read_tile(abi.PT_TILE_ACCUMULATION).tobytes()

    def refused(made, text):
        with pytest.raises(pt.PathTracerError) as e:
            tr.apply_updates(made[0])
        assert e.value.code == abi.PT_ERR_INVALID_ARG and text in e.value.message, e.value.message

    places = {0, triangles - 1} | {triangles * t // 16 + d for t in (1, 7, 15) for d in (-1, 0) if triangles >= 64}
    for at in sorted(places):
        refused(upload(base, triangles, nodes, material_at=at), "material index outside")
    made = upload(base, triangles, nodes)
    made[2]["left_first"][-1] += 1
    refused(made, "leaf triangle range")
    made = upload(base, triangles, nodes, material_at=triangles // 2)
    made[2]["left_first"][-1] += 1
    refused(made, "material index outside")
    refused(upload(base, triangles, nodes, alias=256 * 128), "skybox alias index")
    tr.set_tile((32, 32), (0, 0), (32, 32))
    tr.trace(1)
    assert tr.read_tile(abi.PT_TILE_ACCUMULATION).tobytes() == want
    made = upload(base, triangles, nodes)
    tr.apply_updates(made[0])
    tr.close()
