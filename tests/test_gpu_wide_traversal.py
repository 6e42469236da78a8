"""Closest hits and occlusion over 8-wide hierarchies of every shape a node can take, against the oracle:
no hierarchy (one primitive), a root of leaves only, full leaves, the first root with internal children;
one instance (entered without an instance level) or several; boxes far from the rays' origins, where the
box test's rounding is largest against its one-grid-step margin."""
import math
import os
import subprocess

import numpy as np
import pytest

from mufflon_b200 import bindings, build, scenes

pytestmark = pytest.mark.gpu


def _lod(n, seed):
    """n primitives in the unit cube: triangles, every fourth a quad, every fifth a sphere."""
    rng = np.random.default_rng(seed)
    tris, quads, spheres, v = [], [], [], []
    for k in range(n):
        c = rng.uniform(-1.0, 1.0, 3)
        a, b = rng.normal(scale=0.25, size=(2, 3))
        if k % 5 == 4:
            spheres.append([*c, float(rng.uniform(0.02, 0.3))])
        elif k % 4 == 3:
            quads.append(range(len(v), len(v) + 4))
            v += [c, c + a, c + a + b, c + b]
        else:
            tris.append(range(len(v), len(v) + 3))
            v += [c, c + a, c + b]
    v = np.array(v, np.float32).reshape(-1, 3)
    nv = len(v)
    return scenes.LodSpec(v, np.tile(np.array([0, 0, 1], np.float32), (nv, 1)), np.zeros((nv, 2), np.float32),
                          np.array([list(t) for t in tris], np.uint32).reshape(-1, 3),
                          np.array([list(q) for q in quads], np.uint32).reshape(-1, 4),
                          np.zeros(len(tris) + len(quads), np.uint16), np.array(spheres, np.float32).reshape(-1, 4),
                          np.zeros(len(spheres), np.uint16), name="prims")


def _spec(n, instances, offset, seed):
    rng = np.random.default_rng(seed + 1)
    w2i = []
    for _ in range(instances):
        q = rng.normal(size=(3, 3))
        rot, _ = np.linalg.qr(q)
        s = float(rng.uniform(0.4, 1.5))
        t = offset + (rng.uniform(-2.0, 2.0, 3) if instances > 1 else np.zeros(3))
        w2i.append(np.concatenate([rot.T / s, (-rot.T / s @ t)[:, None]], 1).astype(np.float32).reshape(12))
    mats = [scenes.MaterialSpec(scenes.MAT_LAMBERT)]
    return scenes.SceneSpec([_lod(n, seed)], np.array(w2i, np.float32), np.zeros(instances, np.uint32), mats,
                            np.array([[0, 5, 0, 1, 1, 1]], np.float32), None, (0.0, 0.0, 4.0), (0.0, 0.0, -1.0),
                            (0.0, 1.0, 0.0), math.radians(40.0), 16, 16, name="wide_shapes")


@pytest.mark.parametrize("instances", [1, 2, 8, 9, 70])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 8, 9, 24, 25, 64, 65, 300])
@pytest.mark.parametrize("offset", [0.0, 700.0])
def test_hits_and_occlusion_bit_exact(dll, oracle, n, instances, offset):
    off = np.array([offset, -0.7 * offset, 0.3 * offset])
    spec = _spec(n, instances, off, 17 * n + instances)
    dll.world_clear_all()
    bindings.load_scene_spec(dll, spec)
    assert dll.render_enable_renderer(0, 0)
    assert dll.renderer_set_parameter_int("Megakernel", 0)
    sc = oracle.OracleScene(spec)
    rng = np.random.default_rng(n)
    m = 4000
    org = rng.normal(size=(m, 3)) * 3.0 + (off if offset == 0.0 else 0.0)
    tgt = off + rng.uniform(-2.5, 2.5, (m, 3))
    d = tgt - org
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    if offset == 0.0:  # axis-aligned rays through the primitives' cube, zero components of either sign
        k = m // 4
        ax = rng.integers(0, 3, k)
        d[:k] = np.where(rng.uniform(size=(k, 3)) < 0.5, 0.0, -0.0)
        d[np.arange(k), ax] = np.where(rng.uniform(size=k) < 0.5, -1.0, 1.0)
        org[:k] = rng.uniform(-1.5, 1.5, (k, 3))
    rays = np.concatenate([org, d], 1).astype(np.float32)
    gt, gi, gp, gs = dll.trace_rays(rays)
    ot, oi, op, os_ = sc.trace_first(rays)
    assert np.array_equal(gi, oi) and np.array_equal(gp, op)
    assert np.array_equal(gt.view(np.uint32), ot.view(np.uint32))
    assert np.array_equal(gs.view(np.uint32), os_.view(np.uint32))
    if n >= 8:
        assert (gi >= 0).any()
    a, b = org.astype(np.float32), (org + d * rng.uniform(0.5, 2.0, (m, 1)) * np.linalg.norm(tgt - org, axis=1, keepdims=True)).astype(np.float32)
    assert np.array_equal(dll.trace_occlusion(a, b), sc.trace_any(a, b))


# Coordinates up to 2^58: the box test's products with a clamped reciprocal direction reach the end of the 32-bit
# range (2^49 grid steps of 2^15 at a reciprocal of 2^64, and above), for the object's level and the instances'.
@pytest.mark.parametrize("exponent", [0, 40, 54, 56, 58])
@pytest.mark.parametrize("instances", [1, 3])
def test_axis_rays_at_any_scale(dll, oracle, exponent, instances):
    size = 2.0 ** exponent
    rng = np.random.default_rng(exponent)
    n = 60
    sph = np.concatenate([rng.uniform(-1.0, 1.0, (n, 3)), rng.uniform(0.05, 0.2, (n, 1))], 1) * size
    lod = scenes.LodSpec(np.zeros((0, 3), np.float32), np.zeros((0, 3), np.float32), np.zeros((0, 2), np.float32),
                         np.zeros((0, 3), np.uint32), np.zeros((0, 4), np.uint32), np.zeros(0, np.uint16),
                         sph.astype(np.float32), np.zeros(n, np.uint16), name="spheres")
    spec = _spec(1, instances, np.zeros(3), 1)
    spec.lods[0] = lod
    spec.world_to_instance = np.tile(np.array(scenes.identity34(), np.float32), (instances, 1))
    spec.world_to_instance[:, 3] = np.arange(instances) * np.float32(0.7 * size)
    dll.world_clear_all()
    bindings.load_scene_spec(dll, spec)
    assert dll.render_enable_renderer(0, 0)
    assert dll.renderer_set_parameter_int("Megakernel", 0)
    sc = oracle.OracleScene(spec)
    m = 3000
    d = np.where(rng.uniform(size=(m, 3)) < 0.5, 0.0, -0.0)
    d[np.arange(m), rng.integers(0, 3, m)] = np.where(rng.uniform(size=m) < 0.5, -1.0, 1.0)
    rays = np.concatenate([rng.uniform(-1.2, 1.2, (m, 3)) * size, d], 1).astype(np.float32)
    tmax = float(8.0 * size)
    gt, gi, gp, gs = dll.trace_rays(rays, tmax=tmax)
    ot, oi, op, _ = sc.trace_first(rays, tmax=tmax)
    assert (oi >= 0).sum() > m // 10
    assert np.array_equal(gi, oi) and np.array_equal(gp, op)
    assert np.array_equal(gt.view(np.uint32), ot.view(np.uint32))


def test_box_reciprocal_is_correctly_rounded(tmp_path):
    """Every float of these exponents, zeros and denormals among them: the bits of the IEEE reciprocal."""
    exe = str(tmp_path / "box_reciprocal")
    source = os.path.join(build.ROOT, "tests", "cpp", "box_reciprocal.cu")
    flags = [f for f in build.NVCC_FLAGS if f not in ("-Xptxas", "-v")]
    subprocess.run([build.NVCC, *flags, source, "-o", exe], check=True, capture_output=True)
    exponents = [-127, -126, -97, -65, -64, -63, -37, -17, -7, -2, -1, 0, 1, 13, 63, 125]
    r = subprocess.run([exe, *map(str, exponents)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0
    assert [int(x) for x in r.stdout.split()] == [0] * len(exponents)


# either side of the single-block sort's capacity, few distinct keys and many
@pytest.mark.parametrize("distinct", [3, 1 << 60])
@pytest.mark.parametrize("n", [31, 257, 2047, 2048, 2049])
def test_short_sorts_are_stable(dll, n, distinct):
    rng = np.random.default_rng(n)
    k = rng.integers(0, distinct, n, dtype=np.uint64)
    v = np.arange(n, dtype=np.int32)
    gk, gv = bindings.sort_pairs(dll, k, v)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(gk, k[order]) and np.array_equal(gv, v[order])


# tiles of 2 048 pairs: full ones, one pair over and one short; digits that all lanes of a warp share, and random ones
@pytest.mark.parametrize("distinct", [2, 1 << 60])
@pytest.mark.parametrize("n", [9 * 2048, 9 * 2048 + 1, 17 * 2048 - 1, 130 * 2048 + 31])
def test_tiled_sorts_are_stable(dll, n, distinct):
    rng = np.random.default_rng(n)
    k = np.sort(rng.integers(0, distinct, n, dtype=np.uint64)) if distinct == 2 else rng.integers(0, distinct, n, dtype=np.uint64)
    v = np.arange(n, dtype=np.int32)
    gk, gv = bindings.sort_pairs(dll, k, v)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(gk, k[order]) and np.array_equal(gv, v[order])
