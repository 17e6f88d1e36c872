"""The first launch on a stream that the caller can queue work on depends on that work in full, not by a programmatic edge
(which waits for the one kernel before it only, and that kernel need not have waited for its own predecessors).

pt_trace_noalloc is captured into the caller's CUDA graph behind a kernel, behind a memset and as the first node;
replays give the bits of pt_trace.  pt_trace makes no programmatic launch on the context's stream."""
import ctypes as C

import numpy as np
import pytest

import pathtracer as pt
import wrapped_library
from pathtracer import abi
from test_zz_no_alloc import device_world

pytestmark = pytest.mark.gpu


class EdgeData(C.Structure):
    _fields_ = [("from_port", C.c_uint8), ("to_port", C.c_uint8), ("type", C.c_uint8), ("reserved", C.c_uint8 * 5)]


def edges_of_first_nodes(cu, graph):
    """Edge data of every edge out of a node that nothing precedes."""
    n = C.c_size_t(0)
    assert cu.cuGraphGetEdges_v2(graph, None, None, None, C.byref(n)) == 0
    a, b, d = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (EdgeData * n.value)()
    assert cu.cuGraphGetEdges_v2(graph, a, b, d, C.byref(n)) == 0
    followers = set(b)
    return [bytes(d[i]) for i in range(n.value) if a[i] not in followers]


@pytest.mark.parametrize("before", ["kernel", "memset", "nothing"])
def test_captured_call(before):
    torch = pytest.importorskip("torch")
    lib = pt.load()
    cu = C.CDLL("libcuda.so.1")
    image, origin, tile, bounces, spp = (96, 96), (16, 24), (64, 48), 6, 2
    world = pt.World.cornell_box()
    world.set_aspect_ratio(1.0)
    updates = world.take_updates()
    tracer = pt.PathTracer(updates, tile)
    tracer.set_max_bounces(bounces)
    tracer.set_tile(image, origin, tile)
    assert tracer.trace(spp) == spp
    want = tracer.read_tile(abi.PT_TILE_ACCUMULATION)
    tracer.close()

    keep = []
    dw = device_world(torch, updates, keep)
    accum = torch.zeros((tile[1], tile[0], 4), dtype=torch.float32, device="cuda")
    out = torch.zeros_like(accum)
    other = torch.zeros(64, dtype=torch.float32, device="cuda")
    params = abi.TraceParameters()
    params.image_size[:] = image
    params.tile_origin[:] = origin
    params.max_bounces = bounces
    err = C.create_string_buffer(256)

    def call(stream):
        rc = lib.pt_trace_noalloc(C.byref(dw), C.byref(params), tile[0], tile[1], spp, accum.data_ptr(), out.data_ptr(),
                                  stream, err, len(err))
        assert rc == abi.PT_OK, err.value

    call(None)  # the first call on a device comes before any capture
    other.add_(1.0)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    handle = C.c_void_p(stream.cuda_stream)
    graph, ready = C.c_void_p(), C.c_void_p()
    with torch.cuda.stream(stream):
        assert cu.cuStreamBeginCapture_v2(handle, 2) == 0  # CU_STREAM_CAPTURE_MODE_RELAXED
        if before == "kernel":
            other.add_(1.0)
        elif before == "memset":
            assert cu.cuMemsetD32Async(C.c_uint64(other.data_ptr()), 0, C.c_size_t(64), handle) == 0
        call(handle)
        assert cu.cuStreamEndCapture(handle, C.byref(graph)) == 0
    if before != "nothing":
        first = edges_of_first_nodes(cu, graph)
        assert first and all(e == bytes(8) for e in first)
    accum.fill_(float("nan"))
    torch.cuda.synchronize()
    assert cu.cuGraphInstantiateWithFlags(C.byref(ready), graph, C.c_ulonglong(0)) == 0
    for _ in range(2):
        assert cu.cuGraphLaunch(ready, handle) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(accum.cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert cu.cuGraphExecDestroy(ready) == 0 and cu.cuGraphDestroy(graph) == 0


def test_no_programmatic_launch_on_the_context_stream(tmp_path):
    wrapped_library.run(wrapped_library.link(tmp_path), """
        world = pt.World.cornell_box()
        u = world.take_updates()
        t = pt.PathTracer(u, (200, 150))
        stream = C.c_void_p()
        t._check(t._lib.pt_get_stream(t._h, C.byref(stream)))
        assert stream.value
        C.c_void_p.in_dll(t._lib, "pt_test_watched_stream").value = stream.value
        for samples in (1, 16):
            assert t.trace(samples) == samples
        t.synchronize()
        assert count("watched_launches").value == 0
        t.trace_recorded(1)  # its later launches follow its own on that stream
        assert count("watched_launches").value > 0
        t.close()
        """)
