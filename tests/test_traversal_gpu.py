"""Traversal edges against the oracle's brute-force scan (gpu-marked): node
boxes at the ends of the byte grid's range (flat, tiny, huge and far-off
meshes, nodes of one to five triangles), and shadow rays through more
transparent surfaces than the kernel's collector holds."""

import math

import numpy as np
import pytest

from _parity import assert_passes_match
from oracle.oracle import OracleFilm
from psycles_b200 import _abi, scenes
from psycles_b200.backend import SampleRange
from psycles_b200.materials import ShaderGraph, diffuse_material

pytestmark = pytest.mark.gpu

PASSES = [_abi.PASS_COMBINED, _abi.PASS_NORMAL, _abi.PASS_ALBEDO, _abi.PASS_SAMPLE_COUNT]


def render_both(backend, scene, spp=4, **settings):
    compiled = backend.compile_scene(scene)
    assert compiled.ok(), compiled.diagnostics
    st = scenes.render_settings(48, 40, **settings)
    session = backend.create_session(compiled.scene, st)
    assert session.render_samples(SampleRange(0, spp, 0, spp)), session.diagnostics
    film = OracleFilm(st)
    film.render(scene.to_desc(), 0, spp, spp, brute_force=True)
    assert_passes_match(session, film, PASSES)
    return session


def pane_scene(panes: int):
    """A floor under a sun and a point lamp with `panes` transparent quads
    between, two of them at one distance."""
    g = ShaderGraph()
    g.set_output(g.transparent_bsdf((0.97, 0.93, 0.9)))
    mats = scenes._materials([diffuse_material((0.7, 0.7, 0.7)), g])
    pos, idx = [], []
    heights = [1.0 + 0.05 * max(k, 1) for k in range(panes)]
    for k, y in enumerate(heights):
        pos += [(-2 + 0.1 * k, y, -2), (-2 + 0.1 * k, y, 2), (2, y, 2), (2, y, -2)]
        idx += [(4 * k, 4 * k + 1, 4 * k + 2), (4 * k, 4 * k + 2, 4 * k + 3)]
    meshes = [scenes.quad((-4, 0, -4), (-4, 0, 4), (4, 0, 4), (4, 0, -4)),
              scenes.Mesh(np.array(pos, np.float32), np.array(idx, np.uint32))]
    lights = [scenes.Light(_abi.LIGHT_DISTANT, (1.0, 1.0, 0.9), 2.0, axis_z=(0.2, -0.95, 0.1), angle=0.02),
              scenes.Light(_abi.LIGHT_POINT, (1.0, 0.9, 0.8), 300.0, position=(0.5, 6.0, 0.0), radius=0.1)]
    cam = scenes.Camera(scenes.look_at((0.0, 0.6, 6.0), (0.0, 0.3, 0.0)), math.radians(45), math.radians(45), 0)
    return scenes.Scene(meshes, [scenes.Instance(0, 0), scenes.Instance(1, 1)], mats, lights, cam,
                        background=(0.05, 0.05, 0.05))


@pytest.mark.parametrize("panes,budget", [(7, 8), (8, 8), (9, 8), (9, 9), (10, 9), (16, 32), (17, 32), (26, 64)])
def test_shadow_rays_through_many_transparent_surfaces(backend, panes, budget):
    render_both(backend, pane_scene(panes), max_bounces=2, transparent_max_bounces=budget)


@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1e-4, 0.0), (1e-3, 50.0), (1e4, -3e4), (1.0, 2e3)])
def test_node_boxes_over_scales_and_offsets(backend, scale, offset):
    """Meshes of one to five triangles (full, partly filled and single-leaf
    nodes), axis-aligned flat ones among them, scaled and moved in object
    space; the camera follows."""
    rng = np.random.default_rng(7)
    mats = scenes._materials([diffuse_material((0.7, 0.6, 0.5)), diffuse_material((0.3, 0.5, 0.8))])
    meshes, instances = [], []
    for n in range(1, 6):
        tri = rng.uniform(-1.0, 1.0, (n, 3, 3))
        if n % 2:
            tri[:, :, n % 3] = 0.25  # flat: no extent on one axis
        tri[:, :, 0] += 2.2 * (n - 3)
        pos = (tri.reshape(-1, 3) * scale + offset).astype(np.float32)
        meshes.append(scenes.Mesh(pos, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)))
        instances.append(scenes.Instance(n - 1, n % 2))
    at = lambda *p: tuple(scale * np.array(p) + offset)
    lights = [scenes.Light(_abi.LIGHT_DISTANT, (1.0, 1.0, 1.0), 2.0, axis_z=(0.3, -0.8, -0.5), angle=0.05)]
    cam = scenes.Camera(scenes.look_at(at(0.4, 0.8, 9.0), at(0.0, 0.0, 0.0)), math.radians(60), math.radians(60), 0,
                        near_clip=1e-4 * scale, far_clip=1e5 * max(scale, 1.0))
    scene = scenes.Scene(meshes, instances, mats, lights, cam, background=(0.4, 0.5, 0.6))
    render_both(backend, scene, max_bounces=3)
