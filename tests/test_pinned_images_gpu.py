"""Images that must not change (gpu-marked): cameras hundreds to thousands of
scene sizes away, where the rounding of the triangle test exceeds the padding of
the boxes and a hit depends on the box test and the order of visits.  The
checksums were recorded with a traversal of float boxes throughout."""

import hashlib
import math

import numpy as np
import pytest

from psycles_b200 import _abi, scenes
from psycles_b200.backend import BatchRenderer, SampleRange

pytestmark = pytest.mark.gpu

PASSES = (_abi.PASS_COMBINED, _abi.PASS_NORMAL, _abi.PASS_ALBEDO)
SCENES = {"box": (lambda: scenes.cornell_box(), 1.5), "small": (lambda: scenes.small_test_scene(seed=3), 6.0),
          "procedural": (lambda: scenes.procedural_scene(seed=3, frequencies=(4, 7, 11, 16)), 30.0),
          "lamps": (lambda: scenes.lamp_scene(seed=3), 8.0), "glass": (lambda: scenes.glass_scene(seed=3), 6.0)}
PINNED = {
    ("box", 1e2, 96): "55b4939d152ef214", ("box", 1e2, 384): "da150701552eae12",
    ("box", 1e4, 96): "e6a61509388f5215", ("box", 1e4, 384): "26d4ba9f705acdd7",
    ("box", 1e5, 96): "740738a39f938e44", ("box", 1e5, 384): "b215e2c5df1a47f0",
    ("glass", 1e2, 96): "0ef2136cfc0eaf7e", ("glass", 1e2, 384): "3559e56a4bcee58a",
    ("glass", 1e4, 96): "236b5d189f19b186", ("glass", 1e4, 384): "ab37e67eeed696d8",
    ("glass", 1e5, 96): "f4cc1bf7538c40b6", ("glass", 1e5, 384): "6c6fcc38fef52ac4",
    ("lamps", 1e2, 96): "bdb11458c1af474b", ("lamps", 1e2, 384): "084e9590fad4aa06",
    ("lamps", 1e4, 96): "206adeca67f46ebf", ("lamps", 1e4, 384): "3d17ca92dcf44275",
    ("lamps", 1e5, 96): "f411be1638ce4b52", ("lamps", 1e5, 384): "d525e3daafc1f31f",
    ("procedural", 1e2, 96): "6eab72b5429e7da6", ("procedural", 1e2, 384): "6f8ffe19aec39389",
    ("procedural", 1e4, 96): "0b8ec5ad26a10071", ("procedural", 1e4, 384): "e4c38b4fa137f045",
    ("procedural", 1e5, 96): "3279d110b23f032f", ("procedural", 1e5, 384): "b8a6fcb17b0e64e0",
    ("small", 1e2, 96): "c72b29caf0d65fe6", ("small", 1e2, 384): "bcdfb9077cf9df07",
    ("small", 1e4, 96): "e93c28a93edcde09", ("small", 1e4, 384): "e6491a94cd4e7cc6",
    ("small", 1e5, 96): "1c3d43e059f76d1c", ("small", 1e5, 384): "d607a114df19ee28",
}


def far_scene(name, distance):
    make, extent = SCENES[name]
    scene = make()
    direction = np.array([0.31, 0.24, 0.92]) / math.sqrt(0.31 ** 2 + 0.24 ** 2 + 0.92 ** 2)
    fov = 2.0 * math.atan(1.0 / distance)
    scene.camera = scenes.Camera(scenes.look_at(tuple(direction * distance * extent), (0.0, 0.3 * extent, 0.0)), fov,
                                 fov, 0, near_clip=1e-3, far_clip=1e9)
    return scene


def checksum(session):
    h = hashlib.sha256()
    for kind in PASSES:
        h.update(np.ascontiguousarray(session.read_pass(kind)).tobytes())
    return h.hexdigest()[:16]


def render(backend, name, distance, size):
    """The checksums of one render taken as it comes, step by step in
    wavefronts (a profiled one), and in a batch."""
    compiled = backend.compile_scene(far_scene(name, distance))
    assert compiled.ok(), compiled.diagnostics
    st = scenes.render_settings(size, size, max_bounces=6, seed=4)
    sums = []
    for way in ("plain", "wavefronts", "batch"):
        session = backend.create_session(compiled.scene, st)
        if way == "batch":
            batch = BatchRenderer(backend.context, path_capacity=1 << 18)
            assert batch.render([(session, SampleRange(0, 4, 0, 4))])
            batch.close()
        else:
            if way == "wavefronts":
                _abi.check(session.lib.psy_session_set_profiling(session.handle, 1))
            assert session.render_samples(SampleRange(0, 4, 0, 4)), session.diagnostics
        sums.append(checksum(session))
    return sums


@pytest.mark.parametrize("size", [96, 384])
@pytest.mark.parametrize("distance", [1e2, 1e4, 1e5])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_far_cameras(backend, name, distance, size):
    assert render(backend, name, distance, size) == [PINNED[name, distance, size]] * 3
