"""The wavefront path tracer's schedule only moves work: with lanes refilled one by one or all at once, few paths
spread over many warps, any hand-over to the path-finishing launch and binned or unbinned queues, the image has
the bits of the single-kernel implementation over the binary hierarchies."""
import numpy as np
import pytest

from mufflon_b200 import bindings, scenes

pytestmark = pytest.mark.gpu

DEFAULTS = {"Seed": 0, "Min. path length": 0, "Max. path length": 16, "NEE count": 1, "RR start depth": 0, "Megakernel": 0,
            "Wavefront bounces": 2, "Tail paths": 98304, "Trace blocks per SM": 6, "Trace refill lanes": 12, "Ray sort bits": 0,
            "Tail cost rule": 1, "Planned tail": 1}


def _image(dll, spec, iterations, **params):
    dll.world_clear_all()
    bindings.load_scene_spec(dll, spec)
    assert dll.render_enable_renderer(0, 0)
    dll.render_enable_render_target("Radiance", False)
    for name, value in {**DEFAULTS, **params}.items():
        assert dll.renderer_set_parameter_int(name, value)
    dll.render_reset()
    for _ in range(iterations):
        dll.render_iterate()
    img = dll.get_target_image("Radiance")
    launches = dll.stage_stats()["launches"]
    for name, value in DEFAULTS.items():
        assert dll.renderer_set_parameter_int(name, value)
    return img, launches


def _same(dll, spec, iterations, schedule, **params):
    """Compares the images; the number of kernel launches of the last iteration."""
    a, launches = _image(dll, spec, iterations, **schedule, **params)
    b, _ = _image(dll, spec, iterations, Megakernel=1, **params)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert b.mean() > 0.0
    return launches


@pytest.mark.parametrize("blocks", [4, 5, 6, 8])
@pytest.mark.parametrize("lanes", [1, 12, 32])
def test_refill(dll, lanes, blocks):
    spec = scenes.instanced_scene(1, num_meshes=3, num_instances=40, num_spheres=200, tri_range=(500, 2000), width=120, height=90)
    _same(dll, spec, 1, {"Trace refill lanes": lanes, "Trace blocks per SM": blocks}, **{"NEE count": 2, "Max. path length": 6})


# images of one path, less than a warp, a partly filled launch, more than the launch holds
@pytest.mark.parametrize("size", [(1, 1), (5, 3), (64, 64), (131, 77), (450, 301)])
@pytest.mark.parametrize("sort_bits", [0, 12])
def test_sizes_and_long_paths(dll, size, sort_bits):
    spec = scenes.cornell_box(3, *size)
    _same(dll, spec, 3, {"Ray sort bits": sort_bits}, **{"NEE count": 3, "Max. path length": 20, "RR start depth": 4, "Seed": 5})


# a planned iteration launches camera, the bounces before the hand-over, its trace, the tail and finalize
def _hand_over(launches):
    assert launches % 2 == 0, launches
    return (launches - 4) // 2


@pytest.mark.parametrize("tail", [0, 1000, 1 << 30])
@pytest.mark.parametrize("bounces", [0, 1, 5])
def test_tail_hand_over(dll, bounces, tail):
    spec = scenes.alpha_cutouts(2, 210, 140)
    launches = _same(dll, spec, 2, {"Wavefront bounces": bounces, "Tail paths": tail, "Tail cost rule": 0},
                     **{"NEE count": 2, "Max. path length": 9})
    if tail == 1 << 30:
        assert _hand_over(launches) == bounces
    elif tail == 1000:
        assert _hand_over(launches) >= max(bounces, 3)  # 29 400 paths: not at once
    else:  # never (camera, nine bounces, finalize), or at a bounce that nothing reaches
        assert launches == 2 + 2 * 9 or _hand_over(launches) > bounces


# decided on the device, without a plan: the same hand-overs inside a schedule of every launch
@pytest.mark.parametrize("tail", [1000, 1 << 30])
@pytest.mark.parametrize("bounces", [0, 1, 5])
def test_unplanned_tail_hand_over(dll, bounces, tail):
    spec = scenes.alpha_cutouts(2, 210, 140)
    launches = _same(dll, spec, 2, {"Wavefront bounces": bounces, "Tail paths": tail, "Tail cost rule": 0, "Planned tail": 0},
                     **{"NEE count": 2, "Max. path length": 9})
    assert launches == 2 + 2 * 9 + max(0, 8 - bounces)


@pytest.mark.parametrize("tail", [0, 98304])
def test_tail_hand_over_by_cost(dll, tail):
    _same(dll, scenes.alpha_cutouts(2, 210, 140), 3, {"Tail paths": tail}, **{"NEE count": 2, "Max. path length": 9})
