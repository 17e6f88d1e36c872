"""Workloads of the path-trace pass that a performance measurement times, each through the public entry points.

listed() names the standing cases, draw(rng) makes one more of the same ranges, prepare(case, seed) builds what a
program holds before the call (scene uploaded, tracer or engine created; the seed places the camera, and seeds the
geometry of the small generated scenes), run(state) is one pass and work(case) the bytes and operations a pass cannot
do without.

Kinds of pass
  frame    an interactive frame: camera update, one trace() call from sample 1, the tone-mapped RGBA8 read back
  tile     a still: set_tile() starts the image anew, trace() calls of at most 16 samples, one buffer read back
  headless render_tiles(): the image in tiles of the command line's default side, tone-mapped
  noalloc  pt_trace_noalloc on the caller's own device buffers and the caller's stream
  update   a scene change: apply_updates() with a full upload, a few samples, the RGBA8 read back
  engine   a batch of requests submitted to the batched engine, polled and read back as the serving loop does
"""
import ctypes as C
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path(__file__).resolve().parent.parent / "path-tracer_gb300")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import pathtracer as pt  # noqa: E402
from pathtracer import abi  # noqa: E402
from pathtracer.engine import Engine  # noqa: E402
from pathtracer.serving import SCENE_SIZES  # noqa: E402

# triangles and BVH nodes of each scene (for work(); nodes of the generated ones to a few percent)
TRIANGLES = {"cornell": (36, 45), "cornell_textured": (36, 45), "10k": (9584, 10869), "10k_blend": (9584, 10869),
             "100k": (101632, 115965), "1M": (1009152, 1138575), "2M": (2096640, 2358439)}
HALF = abi.PT_PRECISION_HALF_ATTRIBUTES | abi.PT_PRECISION_KAHAN
WIDE = abi.PT_PRECISION_COMPRESSED


def listed():
    return [
        # the smallest interactive frame: a viewer's small window on a simple room, one sample, latency counts
        {"name": "frame_cornell_160x120", "kind": "frame", "scene": "cornell", "width": 160, "height": 120,
         "samples": 1, "bounces": 10, "precision": 0},
        # a host application's plug-in that owns all device memory: one small ragged tile of a larger image
        {"name": "noalloc_10k_100x70x16", "kind": "noalloc", "scene": "10k", "width": 100, "height": 70,
         "samples": 16, "bounces": 8, "precision": 0},
        # the small still of the reference's default scene: 256x256, 16 samples, depth 8, the sums read back
        {"name": "tile_cornell_256x256x16", "kind": "tile", "scene": "cornell", "width": 256, "height": 256,
         "samples": 16, "bounces": 8, "precision": 0, "result": abi.PT_TILE_ACCUMULATION},
        # an interactive frame of an ordinary scene: one sample of every pixel of a window
        {"name": "frame_100k_640x360", "kind": "frame", "scene": "100k", "width": 640, "height": 360,
         "samples": 1, "bounces": 10, "precision": 0},
        # the textured room of the precision workload in the compressed form, many samples of few pixels
        {"name": "tile_textured_256x256x128", "kind": "tile", "scene": "cornell_textured", "width": 256,
         "height": 256, "samples": 128, "bounces": 8, "precision": WIDE, "result": abi.PT_TILE_IMAGE},
        # materials with partial coverage: random numbers inside the traversal, shadow rays traced while shading
        {"name": "tile_blend_481x271x8", "kind": "tile", "scene": "10k_blend", "width": 481, "height": 271,
         "samples": 8, "bounces": 10, "precision": 0, "result": abi.PT_TILE_IMAGE},
        # the headless command on a size that its 512-pixel tiles do not divide
        {"name": "headless_100k_1000x700x32", "kind": "headless", "scene": "100k", "width": 1000, "height": 700,
         "samples": 32, "bounces": 10, "precision": 0, "tile": 512},
        # another scene loaded into a running viewer, then its first samples
        {"name": "update_1M_960x540x4", "kind": "update", "scene": "1M", "width": 960, "height": 540,
         "samples": 4, "bounces": 8, "precision": 0},
        # one request of the serving mix's fixed shape on an otherwise idle server
        {"name": "engine_1M_512x512x16", "kind": "engine", "scene": "1M", "jobs": 1, "width": 512, "height": 512,
         "samples": 16, "bounces": 8, "precision": HALF, "mix": 0},
        # a batch of the request mix (sides 64..1024, 1..64 samples, depths 4..12, three scenes at once)
        {"name": "engine_mix_16", "kind": "engine", "scene": "10k,100k,1M", "jobs": 16, "width": 0, "height": 0,
         "samples": 0, "bounces": 0, "precision": HALF, "mix": 5},
        # a still in the compressed form (8-wide BVH) on a large scene
        {"name": "tile_1M_wide_1280x720x16", "kind": "tile", "scene": "1M", "width": 1280, "height": 720,
         "samples": 16, "bounces": 8, "precision": WIDE, "result": abi.PT_TILE_IMAGE},
        # the benchmark's still: 2.1M triangles, full HD, 64 samples, depth 8
        {"name": "tile_2M_1920x1080x64", "kind": "tile", "scene": "2M", "width": 1920, "height": 1080,
         "samples": 64, "bounces": 8, "precision": 0, "result": "display"},
    ]


def _side(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "tile", "tile", "tile", "headless", "noalloc", "noalloc", "update",
                       "engine", "engine"])
    opaque = ["cornell", "10k", "100k", "1M"]
    if kind == "engine" and rng.random() < 0.5:
        case = {"kind": kind, "scene": rng.choice(["10k", "100k", "10k,100k", "10k,100k,1M"]),
                "jobs": rng.randint(2, 24), "width": 0, "height": 0, "samples": 0, "bounces": 0,
                "precision": rng.choice([0, HALF, HALF, WIDE]), "mix": rng.randint(1, 1 << 20)}
        while sum(w * h * s for _, w, h, s, _ in _requests(case)) > 90e6:  # at most the largest listed case
            case["jobs"] = max(2, case["jobs"] - 1) if case["jobs"] > 2 else 2
            case["mix"] += 1
        return case
    if kind == "noalloc":
        samples = rng.choice([1, 2, 4, 7, 16])
        most = 0.95 * 262144 / samples  # what one call accepts
        w = _side(rng, 24, min(400, most / 24))
        h = _side(rng, 24, max(25, min(400, most / w)))
        return {"kind": kind, "scene": rng.choice(["cornell", "10k", "10k_blend", "100k"]), "width": w, "height": h,
                "samples": samples, "bounces": rng.randint(2, 12), "precision": 0}
    low, high = {"frame": (80, 900), "tile": (64, 1100), "headless": (300, 1300), "update": (120, 900),
                 "engine": (64, 1024)}[kind]
    side, aspect = _side(rng, low, high), rng.uniform(1.0, 16.0 / 9.0)
    case = {"kind": kind, "scene": rng.choice(opaque), "width": max(8, int(side * math.sqrt(aspect))),
            "height": max(8, int(side / math.sqrt(aspect))), "samples": 1, "bounces": rng.randint(4, 12),
            "precision": 0}
    if kind == "tile":
        case["scene"] = rng.choice(opaque + ["cornell_textured", "10k_blend"])
        case["samples"] = rng.choice([1, 3, 16, 33, 64])
        case["precision"] = rng.choice([0, 0, HALF, WIDE])
        case["result"] = rng.choice([abi.PT_TILE_IMAGE, abi.PT_TILE_ACCUMULATION, "display"])
    elif kind == "headless":
        case["samples"] = rng.choice([4, 16, 20, 32])
        case["tile"] = rng.choice([256, 512, 512])
    elif kind == "update":
        case["samples"] = rng.choice([1, 4, 8])
    elif kind == "engine":
        case.update(jobs=1, mix=0, samples=rng.choice([1, 4, 16, 64]), precision=rng.choice([0, HALF, HALF, WIDE]))
    while case["width"] * case["height"] * case["samples"] > 60e6:
        case["samples"] = max(1, case["samples"] // 2)
    return case


# ---------------------------------------------------------------- scenes and cameras

_worlds = {}


def _world(scene, seed):
    """(World, full updates) of a scene.  The large generated scenes are one scene file each, loaded once per process;
    the small ones are generated from the seed."""
    key = scene if scene in ("1M", "2M", "cornell", "cornell_textured") else (scene, seed)
    if key in _worlds:
        return _worlds[key]
    if scene == "cornell":
        w = pt.World.cornell_box()
    elif scene == "cornell_textured":
        w = pt.World.cornell_box_textured(1)
    elif scene == "2M":
        w = pt.World.procedural()
    else:
        w = pt.World.procedural(seed=7 if scene == "1M" else 100 + seed % 1000, skybox_width=512, skybox_height=256,
                                non_opaque=int(scene.endswith("_blend")), **SCENE_SIZES[scene.split("_")[0]])
    if scene == "2M":
        w.edit_skybox_average_luminance(1.0)  # both kinds of light are sampled
    made = (w, w.take_updates())
    if isinstance(key, str):
        _worlds[key] = made
    return made


def _camera(scene, world, full, rng, width, height):
    """A camera of this scene drawn from rng (camera edits only: the full upload stays valid)."""
    world.set_aspect_ratio(width / height)
    if scene.startswith("cornell"):
        world.edit_camera(yaw=rng.uniform(-0.1, 0.1), pitch=rng.uniform(-0.08, 0.08))
    elif scene == "2M":
        world.edit_camera(position=(rng.uniform(-0.5, 0.5), 14.0, 20.0), yaw=rng.uniform(-0.05, 0.05), pitch=-0.45,
                          fov=1.2)
    else:
        world.edit_camera(yaw=rng.uniform(-0.6, 0.6), pitch=rng.uniform(-0.5, -0.2))
    u = world.take_updates()
    return abi.Camera.from_buffer_copy((u if u.camera else full).camera.contents)


def _full_with(full, camera):
    u = abi.WorldUpdates.from_buffer_copy(full)
    u.camera = C.pointer(camera)
    return u


def _requests(case):
    """(scene, width, height, samples, bounces) of every job of an engine case."""
    scenes = case["scene"].split(",")
    if not case["mix"]:
        return [(scenes[0], case["width"], case["height"], case["samples"], case["bounces"])] * case["jobs"]
    rng, out = random.Random(case["mix"]), []
    for _ in range(case["jobs"]):
        side, aspect = math.exp(rng.uniform(math.log(64), math.log(1024))), rng.uniform(1.0, 16.0 / 9.0)
        out.append((rng.choice(scenes), max(8, int(side * math.sqrt(aspect))), max(8, int(side / math.sqrt(aspect))),
                    rng.choice([1, 4, 16, 64]), rng.randint(4, 12)))
    return out


# ---------------------------------------------------------------- states

class State:
    """What a program keeps between passes."""

    def __init__(self, case):
        self.case = case
        self.keep = []


def _on_device(state, ptr, nbytes):
    host = np.ctypeslib.as_array(C.cast(ptr, C.POINTER(C.c_uint8)), shape=(max(nbytes, 1),))
    state.keep.append(torch.from_numpy(host.copy()).to("cuda"))
    return state.keep[-1].data_ptr()


def _device_world(state, u):
    s, k, dw = u.scene.contents, u.skybox.contents, abi.DeviceWorld()
    dw.geometries = _on_device(state, s.geometries, 36 * s.triangle_count)
    dw.attributes = _on_device(state, s.attributes, 112 * s.triangle_count)
    dw.triangle_count = s.triangle_count
    dw.materials = _on_device(state, s.materials, 224 * s.material_count)
    dw.material_count = s.material_count
    dw.bvh_nodes = _on_device(state, s.bvh_nodes, 32 * s.node_count)
    dw.node_count = s.node_count
    dw.skybox_rgba = _on_device(state, k.rgba, 16 * k.uniforms.width * k.uniforms.height)
    if k.alias_count:
        dw.skybox_aliases = _on_device(state, k.alias_table, 12 * k.alias_count)
    if u.scene_alias_count:
        dw.scene_aliases = _on_device(state, u.scene_alias_table, 16 * u.scene_alias_count)
    dw.camera = u.camera.contents
    dw.scene_uniforms = u.scene_uniforms.contents
    dw.skybox_uniforms = u.skybox_uniforms.contents
    dw.any_non_opaque = int(any(s.materials[i].alpha_mode != abi.PT_ALPHA_MODE_OPAQUE for i in range(s.material_count)))
    return dw


def prepare(case, seed):
    rng = random.Random(seed * 7919 + 13)
    st = State(case)
    if case["kind"] == "engine":
        jobs = _requests(case)
        worlds = {name: _world(name, seed) for name in case["scene"].split(",")}
        cfg = Engine.tuned_config()
        wave = Engine.SERVING_WAVE_PATHS if case["jobs"] == 1 else cfg["wave_paths"]
        st.engine = Engine(wave_paths=wave, tile_size=cfg["tile_size"], steps_per_refill=cfg["steps_per_refill"],
                           precision=case["precision"], sort_min_hits=cfg["sort_min_hits"],
                           traversal_threads=cfg["traversal_threads"], shade_threads=cfg["shade_threads"])
        ids = {name: st.engine.add_scene(full) for name, (_, full) in worlds.items()}
        st.jobs = [(ids[name], _camera(name, *worlds[name], rng, w, h), w, h, s, b) for name, w, h, s, b in jobs]
        st.keep.append(worlds)
        return st
    w, h = case["width"], case["height"]
    world, full = _world(case["scene"], seed)
    st.keep.append((world, full))
    if case["kind"] == "noalloc":
        # the tile sits inside an image three times its size
        st.image, st.origin = (3 * w, 3 * h), (w + seed % 7, h - seed % 5)
        camera = _camera(case["scene"], world, full, rng, *st.image)
        st.world = _device_world(st, _full_with(full, camera))
        st.params = abi.TraceParameters()
        st.params.image_size[:] = st.image
        st.params.tile_origin[:] = st.origin
        st.params.max_bounces = case["bounces"]
        st.params.sample_count = 0
        st.accum = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")
        st.out = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")
        st.error = C.create_string_buffer(256)
        return st
    camera = _camera(case["scene"], world, full, rng, w, h)
    st.full = _full_with(full, camera)
    st.keep.append(camera)
    tile = case.get("tile", 1 << 20)
    st.tracer = pt.PathTracer(st.full, (min(tile, w), min(tile, h)))
    st.tracer.set_max_bounces(case["bounces"])
    if case["precision"]:
        st.tracer.set_precision(case["precision"])
    if case["kind"] == "frame":
        st.moves = abi.WorldUpdates()
        st.moves.camera = C.pointer(camera)
        st.moves.reset_accumulation = 1
    if case["kind"] == "update":
        st.full.reset_accumulation = 1
    return st


def _trace(tracer, samples):
    left = samples
    while left > 0:
        left -= tracer.trace(left)


def run(st):
    case = st.case
    kind, w, h, samples = case["kind"], case["width"], case["height"], case["samples"]
    if kind == "frame":
        st.tracer.apply_updates(st.moves)
        _trace(st.tracer, samples)
        return st.tracer.display_tile()
    if kind == "tile":
        st.tracer.set_tile((w, h), (0, 0), (w, h))
        _trace(st.tracer, samples)
        return st.tracer.display_tile() if case["result"] == "display" else st.tracer.read_tile(case["result"])
    if kind == "headless":
        return pt.render_tiles(st.tracer, w, h, samples, case["tile"])
    if kind == "update":
        st.tracer.apply_updates(st.full)
        _trace(st.tracer, samples)
        return st.tracer.display_tile()
    if kind == "noalloc":
        rc = pt.load().pt_trace_noalloc(C.byref(st.world), C.byref(st.params), w, h, samples, st.accum.data_ptr(),
                                        st.out.data_ptr(), torch.cuda.current_stream().cuda_stream, st.error, 256)
        if rc != abi.PT_OK:
            raise pt.PathTracerError(rc, st.error.value.decode())
        return {"accumulation": st.accum, "image": st.out}
    ids = [st.engine.submit(*job) for job in st.jobs]
    waiting = set(ids)
    while waiting:
        waiting.difference_update(st.engine.poll(timeout_ms=1))
    images = [st.engine.read(j, job[2], job[3], abi.PT_TILE_IMAGE) for j, job in zip(ids, st.jobs)]
    for j in ids:
        st.engine.release(j)
    return images


def exact(case, seed):
    """None: a 64-bit render of the same paths in plain array code (closest hits over up to 2M triangles, several
    bounces) takes far longer than a measurement allows, and one rounding decides which way a path goes."""
    return None


def work(case):
    """Bytes: the scene's buffers once (or what the rays of a small image can touch) and the result once; an update
    also moves the whole upload.  Operations: per ray about 2 log2(n) node visits of two 20-operation box tests and
    log2(n) / 2 triangle tests of 50, per hit 2000 for the shading (its dielectric estimate draws 16 samples)."""
    jobs = _requests(case) if case["kind"] == "engine" else [(case["scene"], case["width"], case["height"],
                                                              case["samples"], case["bounces"])]
    flops = total = 0.0
    touched = {}
    for name, w, h, samples, bounces in jobs:
        n, nodes = TRIANGLES[name]
        paths = w * h * samples
        rays = paths * (4.9 if name.startswith("cornell") else 3.2) * min(1.0, (bounces + 1) / 5.0)
        flops += rays * (2 * math.log2(n) * 40 + math.log2(n) / 2 * 50 + 0.5 * 2000)
        size = n * (36 + 112) + nodes * 32
        touched[name] = min(size, touched.get(name, 0.0) + rays * 3000)
        if case["kind"] == "update":
            total += size
        whole = case["kind"] in ("frame", "headless", "update") or case.get("result") == "display"
        total += w * h * (4 if whole else 32 if case["kind"] == "noalloc" else 16)
    return {"bytes": total + sum(touched.values()), "flops": flops}
