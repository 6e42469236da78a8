"""Abandoned traversals fail the call instead of returning silently wrong pixels.

Every traversal loop is bounded: a ray that exceeds the step limit (or the
traversal stack) is abandoned and counted. Following the reference's error
convention (interface.cpp:53-83: a failing call returns false and leaves a
message for core_get_dll_error), render_iterate then returns false. The test
forces the exit with a tiny "Traversal step limit" (a bounded-loop exit, not a
fault), checks the failure and its message for each renderer and schedule, and
checks that with the limit back at its default the same instance renders the
oracle's image again.
"""
import numpy as np
import pytest

from mufflon_b200 import bindings, scenes
from test_gpu_wide_traversal import _spec

pytestmark = pytest.mark.gpu


def _iterate_ok(d):
    return d.core.render_iterate(d.muffInst, None, None, None) != 0


@pytest.mark.parametrize("renderer,extra", [(0, {"Megakernel": 0}), (0, {"Megakernel": 1}), (1, {"Megakernel": 0}),
                                            (1, {"Megakernel": 1}), (2, {}), (3, {"Megakernel": 0}), (3, {"Megakernel": 1}),
                                            (4, {})],
                         ids=["pt-wavefront", "pt-megakernel", "lt-stages", "lt-single-kernel", "wireframe", "bpt-stages",
                              "bpt-single-kernel", "vcm"])
def test_step_limit_fails_the_iteration(renderer, extra):
    spec = scenes.displaced_icosphere(0, subdiv=4, width=48, height=27)
    d = bindings.DllInterface()
    try:
        bindings.load_scene_spec(d, spec)
        assert d.render_enable_renderer(renderer, 0)
        for k, v in extra.items():
            assert d.renderer_set_parameter_int(k, v)
        assert d.renderer_set_parameter_int("Traversal step limit", 2)
        assert d.renderer_get_parameter_int("Traversal step limit") == 2
        assert not _iterate_ok(d)
        msg = d.core_get_dll_error()
        assert "traversal abandoned" in msg and "step limit of 2" in msg, msg
        assert d.renderer_set_parameter_int("Traversal step limit", 0)
        assert _iterate_ok(d), d.core_get_dll_error()
        assert d.render_stats()["errors"] == 0
    finally:
        d.close()


def test_default_limit_renders_the_oracle_image_after_a_failure(oracle):
    spec = scenes.cornell_box(1, 64, 64)
    d = bindings.DllInterface()
    try:
        bindings.load_scene_spec(d, spec)
        assert d.render_enable_renderer(0, 0)
        assert d.renderer_set_parameter_int("Max. path length", 8)
        d.render_enable_render_target("Hit ID", False)
        assert d.renderer_set_parameter_int("Traversal step limit", 1)
        assert not _iterate_ok(d)
        assert d.renderer_set_parameter_int("Traversal step limit", 0)  # resets the accumulation
        assert _iterate_ok(d), d.core_get_dll_error()
        img = d.get_target_image("Radiance").copy()
        hid = d.get_target_image("Hit ID").copy()
    finally:
        d.close()
    pt = oracle.OraclePathTracer(oracle.OracleScene(spec), seed=0, max_path=8)
    pt.iterate()
    assert np.array_equal(hid, pt.target("Hit ID"))
    assert np.array_equal(img.view(np.uint32), pt.target("Radiance").view(np.uint32))


def test_batch_with_step_limit_fails():
    spec = scenes.cornell_box(2, 32, 32)
    d = bindings.DllInterface()
    try:
        bindings.load_scene_spec(d, spec)
        assert d.render_enable_renderer(0, 0)
        assert d.renderer_set_parameter_int("Traversal step limit", 1)
        with pytest.raises(bindings.MufflonError, match="traversal abandoned"):
            bindings.render_batch([dict(instance=d, spp=1, max_path=4)])
    finally:
        d.close()


# objects without a hierarchy, of a root with leaves only and of several levels, entered from the instance level's
# nodes or from the stack; one instance is entered without an instance level
@pytest.mark.parametrize("instances,n", [(1, 1), (1, 24), (2, 1), (9, 1), (9, 3), (70, 1), (70, 24)])
@pytest.mark.parametrize("renderer", [1, 3], ids=["lt", "bpt"])
def test_both_schedules_abandon_the_same_rays(renderer, instances, n):
    """The stages trace in voted steps and the single kernels in whole ones; the same limit abandons the same rays."""
    d = bindings.DllInterface()
    try:
        bindings.load_scene_spec(d, _spec(n, instances, np.zeros(3), 5))
        assert d.render_enable_renderer(renderer, 0)
        assert d.renderer_set_parameter_int("Max. path length", 4)
        abandoned = {}
        for kernel in (0, 1):
            assert d.renderer_set_parameter_int("Megakernel", kernel)
            for limit in (1, 2, 3, 5, 8, 13, 21, 34, 55, 89, 4096):
                assert d.renderer_set_parameter_int("Traversal step limit", limit)
                ok = _iterate_ok(d)
                errors = d.render_stats()["errors"]
                assert ok == (errors == 0)
                abandoned.setdefault(limit, []).append(errors)
        assert all(a == b for a, b in abandoned.values()), abandoned
        assert abandoned[4096] == [0, 0]
    finally:
        d.close()


def test_every_instance_counts():
    """A ray through two objects of one triangle takes four steps: the instance level's node, the first object, the
    second one taken from the stack, and that object."""
    tri = scenes.LodSpec(np.array([[-9, -9, 0], [9, -9, 0], [0, 9, 0]], np.float32), np.tile(np.array([0, 0, 1], np.float32), (3, 1)),
                         np.zeros((3, 2), np.float32), np.array([[0, 1, 2]], np.uint32), np.zeros((0, 4), np.uint32),
                         np.zeros(1, np.uint16), np.zeros((0, 4), np.float32), np.zeros(0, np.uint16), name="triangle")
    w2i = np.tile(np.array(scenes.identity34(), np.float32), (2, 1))
    w2i[1, 11] = 1.0  # the second one behind the first
    spec = scenes.SceneSpec([tri], w2i, np.zeros(2, np.uint32), [scenes.MaterialSpec(scenes.MAT_LAMBERT)],
                            np.array([[0, 5, 9, 1, 1, 1]], np.float32), None, (0.0, 0.0, 4.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0),
                            0.3, 16, 16, name="two_triangles")
    d = bindings.DllInterface()
    try:
        bindings.load_scene_spec(d, spec)
        assert d.render_enable_renderer(0, 0)
        assert d.renderer_set_parameter_int("Max. path length", 1)
        for limit in (1, 2, 3):
            assert d.renderer_set_parameter_int("Traversal step limit", limit)
            assert not _iterate_ok(d)
        assert d.renderer_set_parameter_int("Traversal step limit", 4)
        assert _iterate_ok(d), d.core_get_dll_error()
    finally:
        d.close()
