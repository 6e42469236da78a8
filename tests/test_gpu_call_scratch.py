"""Ray queries and gradients share an instance's kept device scratch: calls of growing, shrinking and mixed sizes
give the answers of an instance that has made no other call, and the bounds taken on the device are the host's."""
import numpy as np
import pytest

from mufflon_b200 import bindings, scenes

pytestmark = pytest.mark.gpu


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.normal(size=(n, 3)) * 0.3
    d = rng.normal(size=(n, 3))
    return np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)


def test_mixed_calls(core_lib_path):
    def fresh():
        d = bindings.DllInterface(core_lib_path)
        bindings.load_scene_spec(d, scenes.cornell_box_textured(1, 40, 30, texture_size=16))
        assert d.render_enable_renderer(0, 0)
        assert d.renderer_set_parameter_int("Max. path length", 4)
        assert d.renderer_set_parameter_int("RR start depth", 4)
        return d

    used = fresh()
    grad = np.random.default_rng(3).normal(size=(30, 40, 3)).astype(np.float32)
    for n in (1, 1000, 33, 70001, 5):
        rays = _rays(n, n)
        normals = _rays(n, n + 1)[:, 3:] if n % 2 else None
        a, b = used.trace_rays(rays, geo_normals=normals), fresh().trace_rays(rays, geo_normals=normals)
        assert all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))
        ends = rays[:, :3] + rays[:, 3:]
        assert np.array_equal(used.trace_occlusion(rays[:, :3], ends), fresh().trace_occlusion(rays[:, :3], ends))
        d = fresh()
        g0 = used.albedo_gradient(used.textures[0], 2, grad, (16, 16))[0]
        g1 = d.albedo_gradient(d.textures[0], 2, grad, (16, 16))[0]
        # 32-bit atomic sums in another order: at most 2 * 1200 terms of 2^-24 relative each
        assert np.abs(g0 - g1).max() <= 2400 * 2.0 ** -24 * max(np.abs(g1).max(), 1e-30)
        used.render_reset()
        used.render_iterate()
