"""Calls of the CUDA runtime that a test has refused on the host, after which the next call works, on the work that was
asked for; and the number of graphs that an engine makes."""
import pytest

import wrapped_library

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return wrapped_library.link(tmp_path_factory.mktemp("wrapped"))


def test_a_refused_wave_is_launched_later(library):
    """The items of a wave whose graph could not be made run in a later wave, once, as that wave's kernels need: the
    refused job has coverage materials and more paths than the opaque one that follows it."""
    wrapped_library.run(library, """
        from worlds import non_opaque_world
        worlds = [non_opaque_world(), pt.World.cornell_box()]
        updates = [w.take_updates() for w in worlds]
        sizes = [(300, 217), (40, 30)]
        want = []
        for u, size in zip(updates, sizes):
            t = pt.PathTracer(u, size)
            t.set_kernel(abi.PT_KERNEL_PLAIN)
            t.set_max_bounces(6)
            assert t.trace(8) == 8
            want.append(t.read_tile(abi.PT_TILE_ACCUMULATION).tobytes())
            t.close()
        eng = Engine(wave_paths=1 << 20)
        ids = [eng.add_scene(u) for u in updates]
        cameras = [abi.Camera.from_buffer_copy(u.camera.contents) for u in updates]
        for first in (0, 1):  # again when the graphs are there: nothing is refused, nothing is left of the first
            jobs = []
            for k in (0, 1):
                count("refuse_instantiate").value = 1 if first == k == 0 else 0
                try:
                    jobs.append(eng.submit(ids[k], cameras[k], *sizes[k], 8, 6))
                    assert count("instantiated").value > 0
                except pt.PathTracerError as e:
                    assert first == k == 0 and e.code == abi.PT_ERR_OOM, e
                    jobs.append(1)  # the job is queued all the same
                assert count("refuse_instantiate").value == 0
            eng.wait_idle(timeout_ms=20000)
            for k in (0, 1):
                assert eng.status(jobs[k]) == (abi.PT_JOB_DONE, 8)
                assert eng.read(jobs[k], *sizes[k], abi.PT_TILE_ACCUMULATION).tobytes() == want[k]
        eng.close()
        """)


def test_a_refused_launch_is_reported_once(library):
    """The error of a refused launch is not found again by a later call that is in order."""
    wrapped_library.run(library, """
        world = pt.World.cornell_box()
        u = world.take_updates()
        images = []
        for refused in (0, 1):
            t = pt.PathTracer(u, (48, 32))
            count("refuse_launch").value = refused
            try:
                t.trace(2)
                assert not refused
            except pt.PathTracerError as e:
                assert refused and e.code == abi.PT_ERR_CUDA
                t.apply_updates(u)
                t.set_tile((48, 32), (0, 0), (48, 32))
                t.trace(2)
            images.append(t.read_tile(abi.PT_TILE_ACCUMULATION).tobytes())
            t.close()
        assert images[0] == images[1]
        """)


@pytest.mark.parametrize("precision", ["0", "abi.PT_PRECISION_WIDE_BVH"])
def test_waves_of_equal_launches_share_a_graph(library, precision):
    """Waves that the tail kernel ends are the same launches for every depth beyond its round (0 up to 2^17 paths, 1 up
    to 2^18, 5 up to 2^21), so a depth that was not met before makes no graph."""
    wrapped_library.run(library, f"""
        world = pt.World.cornell_box()
        u = world.take_updates()
        eng = Engine(wave_paths=1 << 22, precision={precision})
        sid = eng.add_scene(u)
        cam = abi.Camera.from_buffer_copy(u.camera.contents)
        made = []
        for size, spp in (((64, 64), 4), ((128, 120), 15), ((300, 200), 16)):
            before = count("instantiated").value
            for depth in (0, 1, 2, 3, 4, 5, 6, 7, 9, 12, 16):
                eng.submit(sid, cam, *size, spp, depth)
                eng.wait_idle(timeout_ms=20000)
            made.append(count("instantiated").value - before)
        assert made == [1, 2, 6], made
        eng.close()
        """)


def test_a_trace_refused_in_its_middle_leaves_nothing_behind(library):
    """Every launch of a group in turn (with the hit sort's, whose counts the next group would find) is refused; the
    call after it gives the image it would have given."""
    wrapped_library.run(library, """
        world = pt.World.cornell_box()
        u = world.take_updates()
        t = pt.PathTracer(u, (640, 640))
        t.set_max_bounces(2)

        def image():
            t.set_tile((640, 640), (0, 0), (640, 640))
            t.trace(4)
            return t.read_tile(abi.PT_TILE_ACCUMULATION).tobytes()

        want, refused = image(), 0
        for first in range(40):
            count("accept_launches").value, count("refuse_launch").value = first, 1
            try:
                assert image() == want
            except pt.PathTracerError as e:
                assert e.code == abi.PT_ERR_CUDA
                refused += 1
            done = count("refuse_launch").value == 1  # the group has fewer launches
            count("accept_launches").value = count("refuse_launch").value = 0
            assert image() == want
            if done:
                break
        assert done and refused >= 12, refused
        t.close()
        """)


def test_a_wave_of_plain_launches_refused_in_its_middle_ends_the_engine(library):
    """Nothing follows the refused launch, and the engine says so from then on."""
    wrapped_library.run(library, """
        world = pt.World.cornell_box()
        u = world.take_updates()
        cam = abi.Camera.from_buffer_copy(u.camera.contents)
        for first in (0, 1, 5):
            eng = Engine(wave_paths=1 << 22, use_graphs=False)
            sid = eng.add_scene(u)
            count("accept_launches").value, count("refuse_launch").value = first, 1
            for attempt in range(2):
                try:
                    eng.submit(sid, cam, 640, 640, 4, 3)
                    assert False
                except pt.PathTracerError as e:
                    assert e.code == abi.PT_ERR_CUDA
            assert count("refuse_launch").value == 0
            eng.close()
        """)
