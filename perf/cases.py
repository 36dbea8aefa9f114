"""What a user of this renderer has it do, as timed cases.

Every case goes through the public front end (psycles_b200.backend): a scene
is compiled once and kept resident, sessions, batches or a server render it,
and the passes are read back as a host program reads them.  The sizes are the
ones of bench.py (headline frame, closed box, many lights, viewports, serving
classes) and of the tests, plus odd ones.

    listed()        the fixed cases
    draw(rng)       one more case of the same ranges
    prepare(c, s)   what a program holds before the call: compiled scene,
                    session, batch or server, made from the seed alone
    run(state)      one pass; returns the passes it read, whole
    exact(c, s)     sample counts; a path-traced image has no value in
                    closed form, so its passes are None
    work(c)         what a pass cannot do without
"""

import functools
import math

import numpy as np

from psycles_b200 import _abi, scenes
from psycles_b200.backend import (BatchRenderer, CudaPathTracerBackend, MemoryOutputSink, PassRequest, RenderServer,
                                  SampleRange)

SCENES = {
    "procedural": scenes.procedural_scene,   # 64 instances, 1M triangles, 32 mixed materials, 24 lamps
    "many_light": scenes.many_light_scene,   # 10k emissive triangles
    "box": lambda seed: scenes.cornell_box(),
    "lamps": scenes.lamp_scene,              # lamps in view, transparent pane
    "glossy": scenes.glossy_scene,
    "glass": scenes.glass_scene,
    "values": scenes.value_graph_scene,      # materials linked to value nodes
}
TRIANGLES = {"procedural": 997920, "many_light": 12402, "box": 24, "lamps": 52, "glossy": 580, "glass": 580,
             "values": 580}
COMBINED = [PassRequest(_abi.PASS_COMBINED, "Combined")]
VIEW_SIZES = [(128, 128), (353, 211), (512, 512), (256, 256), (1024, 768), (641, 479), (1920, 1080)]
SERVED_SIZES = [(256, 256), (512, 512), (1024, 768), (640, 360)]


def case(kind, scene, width, height, spp, bounces, **more):
    return dict({"kind": kind, "scene": scene, "width": width, "height": height, "spp": spp, "bounces": bounces},
                **more)


def listed():
    named = {
        # A viewport whose camera moves: one small preview, one sample, the
        # Combined pass.  Launches and host work are most of it.
        "viewport_128": case("viewport", "procedural", 128, 128, 1, 8),
        # Look development: one parameter-only edit, then a few samples of
        # the image over.
        "edit_512": case("edit", "values", 512, 512, 4, 6),
        # The closed box of the small benchmark configuration, every pass.
        "box_256": case("frame", "box", 256, 256, 16, 4),
        # A row bucket of a larger frame at an odd offset, lamps in view.
        "lamps_window": case("frame", "lamps", 1919, 1079, 16, 5, x=301, y=407, w=701, h=203),
        # Dielectric and glossy materials: odd sizes, flat lights and the
        # light tree.
        "glass_odd": case("frame", "glass", 853, 479, 9, 8),
        "glossy_tree": case("frame", "glossy", 960, 540, 16, 6, tree=1),
        # A progressive render: four sample ranges, every pass after each.
        "progressive_720p": case("frame", "procedural", 1280, 720, 8, 8, ranges=4),
        # The many-light configuration: 10k emitters through the light tree.
        "many_light_720p": case("frame", "many_light", 1280, 720, 32, 6, tree=1),
        # The headline frame.
        "frame_1080p": case("frame", "procedural", 1920, 1080, 64, 8),
        # Sixteen viewports of one scene, uneven sizes, in shared wavefronts.
        "viewports_16": case("batch", "procedural", 0, 0, 16, 8, views=16),
        # Jobs of several sizes over two resident scenes through the render
        # server, a parameter edit before and amid them.
        "serve_12": case("serve", "procedural", 0, 0, 32, 8, views=12),
        # Opening a scene: compile, one sample at full size, every pass.
        "open_1080p": case("open", "procedural", 1920, 1080, 1, 8),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _spread(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["viewport", "edit", "frame", "frame", "frame", "frame", "batch", "serve", "open"])
    scene = "procedural" if kind in ("batch", "serve", "open") else rng.choice(sorted(SCENES))
    width = _spread(rng, 96, 1920)
    height = max(64, int(width * rng.uniform(0.4, 1.0)))
    bounces = rng.randint(3, 9)
    spp = {"viewport": 4, "edit": 16, "frame": 64, "batch": 16, "serve": 32, "open": 4}[kind]
    spp = _spread(rng, 1, max(1, min(spp, 40_000_000 // (width * height))))
    c = case(kind, scene, width, height, spp, bounces)
    if kind in ("batch", "serve"):
        c.update(width=0, height=0, views=rng.randint(2, 14))
    if kind == "frame":
        c["tree"] = rng.choice([0, 0, 1])
        if rng.random() < 0.25:
            c["ranges"] = rng.randint(1, 3)
        elif rng.random() < 0.3:
            w, h = rng.randint(32, width), rng.randint(32, height)
            c.update(w=w, h=h, x=rng.randint(0, width - w), y=rng.randint(0, height - h))
    return c


def _views(c):
    """(width, height, samples) of each job of a batched or served case."""
    sizes = VIEW_SIZES if c["kind"] == "batch" else SERVED_SIZES
    return [(*sizes[k % len(sizes)], 1 + (7 * k + c["spp"] - 1) % c["spp"]) for k in range(c["views"])]


def _window(c):
    return c.get("w", c["width"]), c.get("h", c["height"])


@functools.lru_cache(maxsize=4)
def _scene(name, seed):
    return SCENES[name](seed)


def _settings(c, seed, width, height):
    more = {}
    if "w" in c:
        more = {"window_x": c["x"], "window_y": c["y"], "window_width": c["w"], "window_height": c["h"]}
    return scenes.render_settings(width, height, max_bounces=c["bounces"], seed=seed % 65536,
                                  use_light_tree=c.get("tree", 0), **more)


def _camera(rng):
    eye = (rng.uniform(-14, 14), rng.uniform(2, 10), rng.uniform(12, 24))
    target = (rng.uniform(-3, 3), 2.0, rng.uniform(-3, 3))
    return scenes.Camera(scenes.look_at(eye, target), math.radians(45), math.radians(45), 0)


def _edit(rng, scene):
    """A parameter-only edit: other colours and factors in one material."""
    m = int(rng.integers(0, len(scene.materials)))
    block = scene.materials[m].parameters
    return m, rng.uniform(0.1, 0.9, block.scalars.shape), rng.uniform(0.05, 0.95, block.vectors.shape)


def prepare(c, seed):
    rng = np.random.default_rng(seed)
    scene = _scene(c["scene"], seed)
    backend = CudaPathTracerBackend(0)
    if c["kind"] == "open":
        return {"case": c, "backend": backend, "scene": scene,
                "settings": _settings(c, seed, c["width"], c["height"])}
    state = {"case": c}
    if c["kind"] == "serve":
        state["server"] = RenderServer(backend.context)
    elif c["kind"] == "batch":
        state["batch"] = BatchRenderer(backend.context)
    compiled = backend.compile_scene(scene)
    assert compiled.ok(), compiled.diagnostics
    state["scene"] = compiled.scene
    if c["kind"] == "serve":
        other = backend.compile_scene(scenes.procedural_scene(seed + 1, (10, 18, 27), 4))
        assert other.ok(), other.diagnostics
        state["scenes"] = [compiled.scene, other.scene]
        state["edits"] = [_edit(rng, scene)]
        m, scalars, vectors = state["edits"][0]
        state["edits"].append((m, scalars * 0.5, vectors * 0.5))
        state["jobs"] = [(_settings(c, seed + k, w, h), spp, _camera(rng)) for k, (w, h, spp) in enumerate(_views(c))]
    elif c["kind"] == "batch":
        state["jobs"] = [(backend.create_session(compiled.scene, _settings(c, seed + k, w, h), COMBINED), spp,
                          _camera(rng)) for k, (w, h, spp) in enumerate(_views(c))]
    else:
        settings = _settings(c, seed, c["width"], c["height"])
        passes = None if c["kind"] == "frame" else COMBINED
        state["settings"] = settings
        state["session"] = backend.create_session(compiled.scene, settings, passes)
        state["camera"] = _camera(rng)
        state["edit"] = _edit(rng, scene)
    return state


def _pixels(sink):
    return [sink.tiles[k].pixels for k in sorted(sink.tiles)]


def run(state):
    c = state["case"]
    spp = c["spp"]
    if c["kind"] == "serve":
        server, jobs = state["server"], []
        for k, (settings, samples, camera) in enumerate(state["jobs"]):
            if k == 0 or k == len(state["jobs"]) // 2:
                server.rebind_parameters(state["scenes"][0], *state["edits"][0 if k == 0 else 1])
            jobs.append(server.submit(state["scenes"][k % 2], settings, samples, camera))
        images = []
        for job, (settings, _, _) in zip(jobs, state["jobs"]):
            assert server.wait(job) == _abi.PSY_OK
            images.append(server.read_pass(job, _abi.PASS_COMBINED, settings.full_width, settings.full_height))
            server.release(job)
        return images
    if c["kind"] == "batch":
        for session, _, camera in state["jobs"]:
            session.set_camera(camera)
        assert state["batch"].render([(s, SampleRange(0, n, 0, n)) for s, n, _ in state["jobs"]])
        return [s.read_pass(_abi.PASS_COMBINED) for s, _, _ in state["jobs"]]
    sink = MemoryOutputSink()
    if c["kind"] == "open":
        compiled = state["backend"].compile_scene(state["scene"])
        session = state["backend"].create_session(compiled.scene, state["settings"])
        assert session.render_samples(SampleRange(0, spp, 0, spp), sink), session.diagnostics
        session.close()
        compiled.scene.close()
        return _pixels(sink)
    session = state["session"]
    if c["kind"] == "viewport":
        session.set_camera(state["camera"])
    else:
        if c["kind"] == "edit":
            state["scene"].rebind_parameters(*state["edit"])
        session.reset(state["settings"])
    first, step = 0, -(-spp // c.get("ranges", 1))
    while first < spp:
        count = min(step, spp - first)
        assert session.render_samples(SampleRange(first, count, 0, spp), sink), session.diagnostics
        first += count
    return _pixels(sink)


def exact(c, seed):
    if c["kind"] not in ("frame", "open"):
        return None
    w, h = _window(c)
    # the passes in the order of their kinds; the last is the sample count
    return [None] * 5 + [np.full((h, w, 1), float(c["spp"]))]


def work(c):
    """Bytes: the scene's triangles (vertices and normals) read once and the
    passes read back written once.  Operations: per sample about three rays
    (camera, scattered, towards a light), each one descent of a four-wide
    hierarchy (six fused operations a box) to one triangle test, and one
    surface evaluation."""
    jobs = _views(c) if "views" in c else [(*_window(c), c["spp"])]
    pixels = sum(w * h for w, h, _ in jobs)
    samples = sum(w * h * n for w, h, n in jobs)
    every = c["kind"] in ("frame", "open")
    triangles = TRIANGLES[c["scene"]]
    levels = max(1, math.ceil(math.log(triangles, 4)))
    return {"bytes": triangles * 72 + pixels * (84 if every else 16) * c.get("ranges", 1),
            "flops": samples * 3 * (levels * 4 * 12 + 75 + 100)}
