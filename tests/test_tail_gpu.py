"""Short queues finish in one kernel (k_tail): a render takes the same passes
and counts the same rays as one that takes every step as a wavefront (a
profiled render), at path counts around the limit below which a whole render
goes there, and in batches (gpu-marked)."""

import numpy as np
import pytest

from psycles_b200 import _abi, scenes
from psycles_b200.backend import BatchRenderer, SampleRange

pytestmark = pytest.mark.gpu

PASSES = [_abi.PASS_COMBINED, _abi.PASS_NORMAL, _abi.PASS_ALBEDO, _abi.PASS_SAMPLE_COUNT]
SCENES = {"small": scenes.small_test_scene, "glass": scenes.glass_scene, "lamps": scenes.lamp_scene,
          "values": scenes.value_graph_scene}


def passes(session):
    return [session.read_pass(k).view(np.uint32) for k in PASSES]


@pytest.mark.parametrize("name,width,height,spp,tree", [
    ("small", 1, 1, 1, 0), ("small", 33, 3, 1, 0), ("glass", 255, 257, 1, 0), ("small", 256, 256, 1, 1),
    ("lamps", 65537, 1, 1, 0), ("values", 331, 199, 3, 0), ("glass", 160, 120, 9, 1),
    ("small", 160, 128, 1, 0), ("lamps", 20479, 1, 1, 1), ("glass", 20480, 1, 1, 0), ("values", 143, 143, 1, 0)])
def test_tail_equals_wavefronts(backend, name, width, height, spp, tree):
    compiled = backend.compile_scene(SCENES[name](seed=5)).scene
    st = scenes.render_settings(width, height, max_bounces=7, use_light_tree=tree, seed=3)
    plain = backend.create_session(compiled, st)
    assert plain.render_samples(SampleRange(0, spp, 0, spp)), plain.diagnostics
    waves = backend.create_session(compiled, st)
    _abi.check(waves.lib.psy_session_set_profiling(waves.handle, 1))
    assert waves.render_samples(SampleRange(0, spp, 0, spp)), waves.diagnostics
    for a, b in zip(passes(plain), passes(waves)):
        assert np.array_equal(a, b)
    sa, sb = plain.stats(), waves.stats()
    assert (sa.closest_rays, sa.shadow_rays) == (sb.closest_rays, sb.shadow_rays)


@pytest.mark.parametrize("capacity", [4000, 100000])
def test_batched_tail_equals_wavefronts(backend, capacity):
    compiled = [backend.compile_scene(SCENES[n](seed=2)).scene for n in ("small", "glass")]
    work, references = [], []
    for k in range(4):
        st = scenes.render_settings(61 + 9 * k, 47, max_bounces=4 + k, seed=k, use_light_tree=k // 2)
        ref = backend.create_session(compiled[k % 2], st)
        _abi.check(ref.lib.psy_session_set_profiling(ref.handle, 1))
        assert ref.render_samples(SampleRange(0, 5, 0, 5))
        references.append(passes(ref))
        work.append((backend.create_session(compiled[k % 2], st), SampleRange(0, 5, 0, 5)))
    batch = BatchRenderer(backend.context, path_capacity=capacity)
    assert batch.render(work), work[0][0].diagnostics
    for (session, _), ref in zip(work, references):
        for a, b in zip(passes(session), ref):
            assert np.array_equal(a, b)
    batch.close()
