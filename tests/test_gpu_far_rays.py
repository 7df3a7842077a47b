"""Rays from far outside a scene: closest hits are the smallest (distance,
instance, triangle) over all triangles, bit for bit, and any hit agrees, also
where the rounding of the world coordinates is larger than the triangles; and
scenes far from the origin."""
import ctypes as C

import numpy as np
import pytest

import bevy_penumbra_b200 as bp
import oracle
from bevy_penumbra_b200 import scenes
from tests.helpers import EMPTY, empty_device, from_device, quat_xyz, to_device

pytestmark = pytest.mark.gpu

SIDE = 256  # quads of the grid's edge


def grid_scene(at=(0.0, 0.0, 0.0), alone=False):
    """A bumped grid of 2 units (131,072 triangles), rotated, at a place;
    `alone`, or with seven small quads beside it (few turned instances keep the
    two-level walk, these take the flattened tree)."""
    u = np.linspace(-1.0, 1.0, SIDE + 1)
    x, y = np.meshgrid(u, u, indexing="ij")
    v = np.stack([x, y, 0.1 * np.sin(5 * x) * np.cos(4 * y)], -1).reshape(-1, 3).astype(np.float32)
    i, j = (a.reshape(-1) for a in np.meshgrid(np.arange(SIDE), np.arange(SIDE), indexing="ij"))
    a = i * (SIDE + 1) + j
    tri = np.concatenate([np.stack([a, a + SIDE + 1, a + SIDE + 2], 1), np.stack([a, a + SIDE + 2, a + 1], 1)])
    desc = scenes.SceneDesc(name="grid")
    mat = desc.add_material(scenes.material_words((0.5, 0.5, 0.5)))
    m = np.zeros((3, 4), np.float32)
    m[:, :3] = quat_xyz(0.5, 0.3, 0.0)
    m[:, 3] = at
    desc.add_instance(desc.add_mesh(scenes.Mesh(v, tri.astype(np.uint32))), m, flags=8, material=mat)
    small = desc.add_mesh(scenes.quad((-0.02, -0.02, 0), (0.02, -0.02, 0), (0.02, 0.02, 0), (-0.02, 0.02, 0)))
    for k in range(0 if alone else 7):
        p = m.copy()
        p[:, 3] += m[:, :3] @ np.float32([0.9, -0.9 + 0.3 * k, -0.05])
        desc.add_instance(small, p, flags=8, material=mat)
    return bp.PackedScene.from_desc(desc), m


def rays_to(m, distance, count, seed):
    """Rays from `distance` away to points well inside the grid, along the
    world axes and oblique."""
    rng = np.random.default_rng(seed)
    p = np.concatenate([rng.uniform(-0.6, 0.6, (count, 2)), np.zeros((count, 1))], 1)
    target = p @ m[:, :3].astype(np.float64).T + m[:, 3]
    d = rng.normal(size=(count, 3))
    d[: count // 2] = np.eye(3)[rng.integers(0, 3, count // 2)]
    d *= np.sign(d @ m[:, :3].astype(np.float64)[:, 2])[:, None]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros(count, dtype=bp.RAY_DTYPE)
    rays["origin"] = target - d * distance
    rays["direction"] = d
    rays["limit"] = 1e20
    return rays


def brute(packed, rays):
    scene = oracle.OracleScene.from_packed(packed)
    hits = np.zeros(len(rays), dtype=bp.HIT_DTYPE)
    for k, r in enumerate(rays):
        o, d = np.ascontiguousarray(r["origin"]), np.ascontiguousarray(r["direction"])
        oracle.lib().orc_brute_closest(scene.handle, o.ctypes.data, d.ctypes.data, C.c_float(0.0), C.c_float(1e20),
                                       hits[k:k + 1].ctypes.data)
    return hits


def check(packed, rays):
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed)
    want = brute(packed, rays)
    assert np.mean(want["triangle"] != EMPTY) > 0.9
    d_rays, d_hits = to_device(rays), empty_device(len(rays) * bp.HIT_DTYPE.itemsize)
    for any_hit in (False, True):
        bp.trace_rays(ctx, scene, d_rays.data_ptr(), len(rays), d_hits.data_ptr(), any_hit=any_hit)
        got = from_device(d_hits, bp.HIT_DTYPE, (len(rays),))
        np.testing.assert_array_equal(got["errors"], np.zeros_like(got["errors"]))
        np.testing.assert_array_equal(got["triangle"] != EMPTY, want["triangle"] != EMPTY)
        if not any_hit:
            hit = want["triangle"] != EMPTY
            np.testing.assert_array_equal(got["triangle"], want["triangle"])
            np.testing.assert_array_equal(got["distance"].view(np.uint32), want["distance"].view(np.uint32))
            np.testing.assert_array_equal(got["barycentric"][hit], want["barycentric"][hit])
    # The radiance call's distances are those of the closest hits.
    d_out = empty_device(len(rays) * 16)
    settings = bp.RadianceCascades().sanitized()
    bp.interval_radiance(ctx, scene, settings, d_rays.data_ptr(), len(rays), d_out.data_ptr())
    hit = want["triangle"] != EMPTY
    np.testing.assert_array_equal(from_device(d_out, np.float32, (len(rays), 4))[hit, 3], want["distance"][hit])


@pytest.mark.parametrize("alone", [False, True])
@pytest.mark.parametrize("distance", [3.0, 10.0, 20.0, 60.0, 130.0, 2e3, 2e4, 2e5])
def test_rays_from_outside(distance, alone):
    packed, m = grid_scene(alone=alone)
    check(packed, rays_to(m, distance, 700, int(distance)))


@pytest.mark.parametrize("place", [60.0, 300.0, 1e4, 1e5])
def test_scene_far_from_the_origin(place):
    packed, m = grid_scene((place, -0.5 * place, 0.25 * place))
    check(packed, rays_to(m, 3.0, 400, int(place)))


def test_refit_far_from_the_origin_and_back():
    """A refit that takes a detailed scene far from the origin leaves the
    flattened tree, one that brings it back returns to it."""
    near, m0 = grid_scene()
    far, m1 = grid_scene((1e5, 0.0, -2e4))
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, near)
    for packed, m in ((far, m1), (near, m0)):
        base = int(packed.scene_words[0, 1])
        rows = packed.scene_words.view(np.float32)
        caller = {int(c): rows[base + 9 * i + 3:base + 9 * i + 6] for i, c in enumerate(packed.instance_order)}
        scene.refit(np.stack([caller[int(c)] for c in near.instance_order]))
        rays = rays_to(m, 3.0, 300, 8)
        d_rays, d_hits = to_device(rays), empty_device(len(rays) * bp.HIT_DTYPE.itemsize)
        bp.trace_rays(ctx, scene, d_rays.data_ptr(), len(rays), d_hits.data_ptr())
        got, want = from_device(d_hits, bp.HIT_DTYPE, (len(rays),)), brute(packed, rays)
        np.testing.assert_array_equal(got["errors"], 0)
        np.testing.assert_array_equal(got["triangle"], want["triangle"])
        np.testing.assert_array_equal(got["distance"].view(np.uint32), want["distance"].view(np.uint32))
