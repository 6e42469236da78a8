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


# around the size from which bounds are taken on the device; spheres beyond the vertices; exact zeros, whose sign
# the host's order decides
@pytest.mark.parametrize("n", [8000, 8192, 9001, 40000])
@pytest.mark.parametrize("zeros", [False, True])
def test_device_bounds(dll, n, zeros):
    rng = np.random.default_rng(n)
    nt = n // 3
    v = rng.uniform(-3.0, 5.0, (3 * nt, 3)).astype(np.float32)
    if zeros:
        v = np.abs(v)
        v[rng.integers(0, len(v), 40), 1] = np.where(rng.uniform(size=40) < 0.5, np.float32(0.0), np.float32(-0.0))
    sph = np.concatenate([rng.uniform(0.5, 6.0, (n - 3 * nt + 50, 3)), rng.uniform(0.01, 0.4, (n - 3 * nt + 50, 1))], 1).astype(np.float32)
    lod = scenes.LodSpec(v, np.tile(np.array([0, 0, 1], np.float32), (len(v), 1)), np.zeros((len(v), 2), np.float32),
                         np.arange(3 * nt, dtype=np.uint32).reshape(nt, 3), np.zeros((0, 4), np.uint32), np.zeros(nt, np.uint16),
                         sph, np.zeros(len(sph), np.uint16), name="cloud")
    spec = scenes.SceneSpec([lod], np.array([scenes.identity34()], np.float32), np.zeros(1, np.uint32),
                            [scenes.MaterialSpec(scenes.MAT_LAMBERT)], np.array([[0, 9, 0, 1, 1, 1]], np.float32), None,
                            (0.0, 0.0, 9.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0), 0.7, 16, 16, name="cloud")
    dll.world_clear_all()
    bindings.load_scene_spec(dll, spec)
    nodes, prims, internal = dll.get_bvh(0)
    _, _, want, want_prims, want_internal, _ = bindings.lbvh_build(dll, lod)  # with the host's bounds
    assert internal == want_internal and np.array_equal(prims, want_prims)
    assert np.array_equal(nodes.view(np.uint32), want.view(np.uint32))
