"""Calls in a row, whose groups overlap, and calls after a synchronisation, whose groups run alone: on both sides of the
sizes at which a hit's lanes share its shading (2^15 paths beside other groups, 2^19 with coverage materials, 2^20
alone), in every form.  Against the plain kernel, bit for bit."""
import pytest

import pathtracer as pt
from pathtracer import abi
from worlds import non_opaque_world

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def worlds():
    out = {"room": pt.World.cornell_box(), "coverage": non_opaque_world()}
    return {name: (w, w.take_updates()) for name, w in out.items()}


@pytest.mark.parametrize("synchronised", [False, True])
@pytest.mark.parametrize("scene,precision,size,spp", [
    ("room", 0, (128, 16), 16), ("room", 0, (129, 16), 16), ("room", abi.PT_PRECISION_WIDE_BVH, (129, 16), 16),
    ("coverage", 0, (256, 128), 16), ("coverage", 0, (257, 128), 16), ("room", 0, (256, 256), 16), ("room", 0, (257, 256), 16)])
def test_equal_to_the_plain_kernel(worlds, scene, precision, size, spp, synchronised):
    out = []
    for kernel in (abi.PT_KERNEL_PLAIN, abi.PT_KERNEL_WAVEFRONT):
        t = pt.PathTracer(worlds[scene][1], size)
        t.set_kernel(kernel)
        if kernel == abi.PT_KERNEL_WAVEFRONT and precision:
            t.set_precision(precision)
        t.set_max_bounces(6)
        for k in range(5):
            assert t.trace(spp) == spp
            if synchronised and k % 2:
                t.synchronize()
        out.append(t.read_tile(abi.PT_TILE_ACCUMULATION).tobytes())
        t.close()
    assert out[0] == out[1]
