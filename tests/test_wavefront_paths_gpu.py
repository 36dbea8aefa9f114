"""Short renders step by step in wavefronts (gpu-marked).  A render of fewer than
20 Ki paths otherwise ends in one kernel, which most GPU tests' renders would
do as a whole; with sort thresholds of one path every queue is traced, sorted,
shaded and shadowed by the wavefront kernels.  Other files' tests run here
again in that way: single sessions against the oracle, batches and the render
server against sessions alone."""

import numpy as np
import pytest
import torch

import test_batch
import test_camera
import test_glass_gpu
import test_glossy_gpu
import test_gpu_parity
import test_lamp_events
import test_light_tree
import test_server
import test_stack_bound
import test_tail_gpu
import test_traversal_gpu
import test_value_stream_gpu
from psycles_b200 import autotune, scenes
from psycles_b200.backend import BatchRenderer, SampleRange

pytestmark = pytest.mark.gpu

SORTED = {"sort_threshold": 1, "shadow_sort_threshold": 1, "ray_sort_threshold": 1}
# a limit of one path alone: the shading sort off, shadow queues sorted
PLAIN = {"sort_threshold": 0, "shadow_sort_threshold": 1, "ray_sort_threshold": 0}
PANES = [(7, 8), (9, 8), (10, 9), (17, 32), (26, 64)]

CASES = {
    "box": (test_gpu_parity.test_cornell_box_passes_match_oracle,),
    "small": (test_gpu_parity.test_small_scene_all_closures_and_lights,),
    "lamps": (test_lamp_events.test_lamp_scene_passes_match_oracle,),
    "glossy": (test_glossy_gpu.test_glossy_scene_matches_oracle, 0),
    "glossy tree": (test_glossy_gpu.test_glossy_scene_matches_oracle, 1),
    "glass": (test_glass_gpu.test_glass_scene_matches_oracle, 0),
    "glass tree": (test_glass_gpu.test_glass_scene_matches_oracle, 1),
    "values tree": (test_value_stream_gpu.test_value_graph_scene_matches_oracle, 1),
    "small tree": (test_light_tree.test_tree_render_small_scene_matches_oracle,),
    "many lights": (test_light_tree.test_tree_render_many_lights_matches_oracle,),
    "stack bound": (test_stack_bound.test_degenerate_trees_fit_the_stack_and_match_brute_force,),
    "edit": (test_gpu_parity.test_rebind_parameters_equals_recompiled_scene,),
    "batch graph": (test_batch.test_batch_equals_sessions_alone, True),
    "batch": (test_batch.test_batch_equals_sessions_alone, False),
    "batch glossy": (test_glossy_gpu.test_glossy_batched_equals_alone,),
    "batch glass": (test_glass_gpu.test_glass_batched_equals_alone,),
    "batch tree": (test_tail_gpu.test_batched_tail_equals_wavefronts, 4000),
    "server": (test_server.test_jobs_equal_sessions_alone_in_a_mix,),
    "server edits": (test_server.test_parameter_edits_are_ordered_with_jobs,),
    "server tree edits": (test_server.test_emissive_edit_while_a_tree_job_runs,),
    **{f"camera {c}": (test_camera.test_camera_rays_and_passes_match_oracle, c) for c in sorted(test_camera.CASES)},
    **{f"panes {p}": (test_traversal_gpu.test_shadow_rays_through_many_transparent_surfaces, *p) for p in PANES},
}


@pytest.fixture(params=["sorted", "plain"])
def wavefronts(request, backend):
    default = autotune.get_tuning(backend)
    autotune.set_tuning(backend, dict(default, **(SORTED if request.param == "sorted" else PLAIN)))
    yield backend
    autotune.set_tuning(backend, default)


@pytest.mark.parametrize("case", sorted(CASES))
def test_in_wavefronts(wavefronts, case):
    function, *arguments = CASES[case]
    function(wavefronts, *arguments)


@pytest.mark.parametrize("knob", ["sort_threshold", "shadow_sort_threshold", "ray_sort_threshold"])
def test_thresholds_below_the_tail_limit_take_effect(backend, knob):
    """A render of 4800 paths is one launch of the tail kernel by default, and
    takes its steps in wavefronts where a threshold asks for it."""
    default = autotune.get_tuning(backend)
    compiled = backend.compile_scene(scenes.small_test_scene(seed=6)).scene
    launches, images = {}, {}
    try:
        for value in (default[knob], 1, 4800, 4801):
            autotune.set_tuning(backend, dict(default, **{knob: value}))
            session = backend.create_session(compiled, scenes.render_settings(80, 60, max_bounces=5))
            assert session.render_samples(SampleRange(0, 1, 0, 1))
            launches[value], images[value] = session.stats().kernel_launches, session.read_pass(0)
    finally:
        autotune.set_tuning(backend, default)
    assert launches[4801] == launches[default[knob]] < launches[4800] <= launches[1]
    for image in images.values():
        assert np.array_equal(image, images[1])


def count_kernels(work):
    """Kernels of this library that `work` ran, as the CUDA activity records show them."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        work()
        torch.cuda.synchronize()
    return sum("psy::k_" in e.name for e in prof.events())


@pytest.mark.parametrize("tree", [0, 1])
@pytest.mark.parametrize("tuning", [{}, SORTED], ids=["default", "sorted"])
def test_kernel_launch_counts(backend, tuning, tree):
    torch.zeros(1, device="cuda")
    default = autotune.get_tuning(backend)
    compiled = backend.compile_scene(scenes.small_test_scene(seed=6)).scene
    settings = scenes.render_settings(80, 60, max_bounces=5, use_light_tree=tree)
    try:
        autotune.set_tuning(backend, dict(default, **tuning))
        session = backend.create_session(compiled, settings)
        ran = count_kernels(lambda: session.render_samples(SampleRange(0, 1, 0, 4)))
        assert session.stats().kernel_launches == ran
        for graph in (False, True):
            batch = BatchRenderer(backend.context, path_capacity=9000, use_graph=graph)
            ran = count_kernels(lambda: batch.render([(session, SampleRange(1, 3, 0, 4))]))
            assert batch.stats().kernel_launches == ran
            batch.close()
            session = backend.create_session(compiled, settings)
    finally:
        autotune.set_tuning(backend, default)
