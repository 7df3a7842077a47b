"""The flattened tree (world-space copies of the instances' nodes) and the
two-level walk it replaces: both against the oracle, bit for bit, on the poses
that decide between them, and the step budgets of a walk that runs past them."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
import oracle
from bevy_penumbra_b200 import scenes
from tests.helpers import EMPTY, empty_device, from_device, to_device
from tests.test_gpu_radiance import oracle_radiance, random_rays

pytestmark = pytest.mark.gpu


def trace(packed, rays, any_hit=False):
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed)
    d_rays = to_device(rays)
    d_hits = empty_device(len(rays) * bp.HIT_DTYPE.itemsize)
    bp.trace_rays(ctx, scene, d_rays.data_ptr(), len(rays), d_hits.data_ptr(), any_hit=any_hit)
    return from_device(d_hits, bp.HIT_DTYPE, (len(rays),))


def cornell_with(linear, at=(0.2, 0.9, 0.1)):
    """The Cornell box and one cube of a given linear part."""
    desc = scenes.cornell()
    cube = desc.add_mesh(scenes.box_mesh((0.3, 0.3, 0.3)))
    m = np.zeros((3, 4), np.float32)
    m[:, :3] = linear
    m[:, 3] = at
    flags = 8 | (4 if np.linalg.det(np.asarray(linear, np.float64)) < 0 else 0)
    desc.add_instance(cube, m, flags=flags, material=0)
    return bp.PackedScene.from_desc(desc)


POSES = {
    "identity": np.eye(3),
    "rotated": scenes.rotation_y(0.7)[:, :3] @ np.diag((1.0, 2.0, 0.25)),
    "mirrored": np.diag((-1.0, 1.5, 1.0)),
    "thin": np.diag((1e-3, 1.0, 3.0)),
    "sheared": np.array([[1.0, 0.5, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]]),     # still flattened
    "ill-sheared": np.array([[1.0, 9.0, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]]),  # the two-level walk
}


@pytest.mark.parametrize("pose", list(POSES))
def test_hits_and_radiance_match_the_oracle_for_every_pose(pose):
    packed = cornell_with(POSES[pose])
    rays = random_rays(4133, (-0.95, 0.05, -0.95), (0.95, 1.95, 0.95), seed=5)
    rays["direction"][:6] = np.concatenate([np.eye(3), -np.eye(3)]).astype(np.float32)
    rays["direction"][6:9, 1] = 0.0
    rays["limit"][9::4] = 0.4
    rays["tmin"][10::4] = 0.2
    cpu, _ = oracle.OracleScene.from_packed(packed).trace_rays(rays)
    gpu = trace(packed, rays)
    for field in ("triangle", "instance", "errors"):
        np.testing.assert_array_equal(gpu[field], cpu[field], err_msg=field)
    hit = cpu["triangle"] != EMPTY
    np.testing.assert_array_equal(gpu["distance"][hit].view(np.uint32), cpu["distance"][hit].view(np.uint32))
    np.testing.assert_array_equal(gpu["barycentric"][hit], cpu["barycentric"][hit])
    blocked, _ = oracle.OracleScene.from_packed(packed).trace_rays(rays, any_hit=True)
    np.testing.assert_array_equal(trace(packed, rays, True)["triangle"] != EMPTY, blocked["triangle"] != EMPTY)
    settings = bp.RadianceCascades(emissive_samples=8, frame_index=5).sanitized()
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed)
    d_rays, d_out = to_device(rays), empty_device(len(rays) * 16)
    bp.interval_radiance(ctx, scene, settings, d_rays.data_ptr(), len(rays), d_out.data_ptr())
    np.testing.assert_array_equal(from_device(d_out, np.float32, (len(rays), 4)).view(np.uint32),
                                  oracle_radiance(packed, settings, rays).view(np.uint32))


@pytest.mark.parametrize("pose", ["rotated", "ill-sheared"])
def test_refit_moves_between_the_walks(pose):
    """A refit to an ill-conditioned pose leaves the flattened tree, one back
    returns to it; hits are those of the scene packed at the pose."""
    start = cornell_with(POSES["rotated" if pose == "ill-sheared" else "ill-sheared"])
    target = cornell_with(POSES[pose])
    rays = random_rays(2049, (-0.95, 0.05, -0.95), (0.95, 1.95, 0.95), seed=9)
    rows = target.scene_words.view(np.float32)
    base = [int(target.scene_words[0, 1]) + 9 * i for i in range(len(target.instance_order))]
    caller = {int(c): rows[b + 3:b + 6] for c, b in zip(target.instance_order, base)}
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, start)
    scene.refit(np.stack([caller[int(c)] for c in start.instance_order]))
    d_rays, d_hits = to_device(rays), empty_device(len(rays) * bp.HIT_DTYPE.itemsize)
    bp.trace_rays(ctx, scene, d_rays.data_ptr(), len(rays), d_hits.data_ptr())
    got, want = from_device(d_hits, bp.HIT_DTYPE, (len(rays),)), trace(target, rays)
    np.testing.assert_array_equal(got["distance"].view(np.uint32), want["distance"].view(np.uint32))
    np.testing.assert_array_equal(got["triangle"] != EMPTY, want["triangle"] != EMPTY)


def comb(one_mesh, teeth=24000):
    """Triangles in a row whose boxes a long ray crosses without meeting a
    triangle, and a wall behind them: as one mesh, or one instance each."""
    desc = scenes.SceneDesc(name="comb")
    mat = desc.add_material(scenes.material_words((0.5, 0.5, 0.5)))
    tooth = np.array([[0, 0, 0], [1, 1, 0], [0, 1, 1]], np.float32)
    if one_mesh:
        v = np.concatenate([tooth + np.float32([0.25 * i, 0, 0]) for i in range(teeth)])
        mesh = desc.add_mesh(scenes.Mesh(v, np.arange(3 * teeth, dtype=np.uint32).reshape(-1, 3)))
        desc.add_instance(mesh, material=mat)
    else:
        mesh = desc.add_mesh(scenes.Mesh(tooth, np.array([[0, 1, 2]], np.uint32)))
        for i in range(teeth):
            m = np.eye(3, 4, dtype=np.float32)
            m[0, 3] = 0.25 * i
            desc.add_instance(mesh, m, material=mat)
    x = 0.25 * teeth + 5.0
    wall = desc.add_mesh(scenes.quad((x, -4, -4), (x, 4, -4), (x, 4, 4), (x, -4, 4)))
    desc.add_instance(wall, material=mat)
    return bp.PackedScene.from_desc(desc)


@pytest.mark.parametrize("one_mesh", [True, False])
def test_step_budgets_are_those_of_the_two_level_walk(one_mesh):
    """A ray along the comb exceeds the 4096-step budget of its walk: the
    instance (then the wall behind is found) or the whole query is abandoned
    as unsupported.  Short rays and rays beside the comb are unaffected."""
    packed = comb(one_mesh)
    rng = np.random.default_rng(3)
    rays = np.zeros(200, dtype=bp.RAY_DTYPE)
    rays["origin"] = np.float32([-1.0, 0.05, 0.95]) + rng.uniform(-0.02, 0.02, (200, 3)).astype(np.float32)
    rays["direction"] = np.float32([1.0, 0.0, 0.0])
    rays["limit"] = 1e20
    rays["limit"][64:128] = rng.uniform(2.0, 60.0, 64)
    rays["origin"][128:, 1] = 2.0
    for any_hit in (False, True):
        cpu, _ = oracle.OracleScene.from_packed(packed).trace_rays(rays, any_hit=any_hit)
        gpu = trace(packed, rays, any_hit)
        np.testing.assert_array_equal(gpu["errors"] & 4, cpu["errors"] & 4)
        np.testing.assert_array_equal(gpu["triangle"] != EMPTY, cpu["triangle"] != EMPTY)
        if not any_hit:
            np.testing.assert_array_equal(gpu["errors"][:64] & 4, np.full(64, 4))
            assert np.all((gpu["triangle"][:64] != EMPTY) == one_mesh) and np.all(gpu["triangle"][128:] != EMPTY)
            hit = cpu["triangle"] != EMPTY
            np.testing.assert_array_equal(gpu["distance"][hit].view(np.uint32), cpu["distance"][hit].view(np.uint32))
