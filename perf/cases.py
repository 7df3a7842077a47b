"""Performance cases of the transport library: the work a host engine has it do.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare(case, seed)`` builds what a host holds before the call
(scene, view, device or host buffers, cache), ``run(state)`` is one pass
through the public entry points, ``work(case)`` the bytes and operations the
pass cannot do without, ``exact(case, seed)`` the outputs in 64 bits where
they have a closed definition.

Scenes, cameras and settings are those of the benchmark and the tests: the
Cornell box, the atrium, the room scenes of the batched workload and the
moving 1,048,576-triangle scene, with the reference's default four cascades or
the benchmark's eight.  A seed moves the camera, the frame index, the rays and
the samples; the scene geometry belongs to the case, as an engine keeps one
scene for many frames.
"""
import functools
import math

import numpy as np
import torch

import bevy_penumbra_b200 as bp
from bevy_penumbra_b200 import scenes

DEVICE = "cuda:0"
FOV = 60.0
EMPTY = -1  # LUX_EMPTY read as int32
DENSE_WIDTH, DENSE_HEIGHT = 320, 240  # pixels the dense case resolves

FRAME = {"kind": "frame", "scene": "room", "triangles": 20000, "width": 320, "height": 180, "stride": 4, "points": 1,
         "rays": 1, "levels": 4, "ratio": 4.0, "samples": 16, "history": True, "host": False, "sort": False,
         "bounce": False, "sky": False, "lights": 0, "lod": False, "moving": False}


def _frame(**fields):
    return dict(FRAME, **fields)


def listed():
    return [
        # A small preview view of the Cornell box with the default settings:
        # some 600 rays, where launches and their gaps are the frame.
        _frame(name="frame_cornell_preview", scene="cornell", triangles=34, width=64, height=48, stride=2, points=1),
        # The default settings (four cascades, one ray per receiver, world
        # history) in the call a host engine makes: host buffers in and out.
        _frame(name="frame_host_360p", scene="atrium", triangles=65536, width=640, height=360, host=True),
        # The benchmark frame: eight cascades, 36 rays per receiver, visibility
        # queries in coherence order, every pixel resolved.
        _frame(name="frame_720p_8level", scene="atrium", triangles=262144, width=1280, height=720, rays=36, levels=8,
               ratio=2.0, sort=True),
        # The largest frame: a million triangles, emitters that move every
        # frame (refit, new emitter records, invalidated history), half of the
        # pixels of each axis resolved.
        _frame(name="frame_1080p_moving", scene="full", triangles=1 << 20, width=1920, height=1080, points=2, rays=36,
               levels=8, ratio=2.0, moving=True),
        # Multi-bounce with the sky cached in the secondary cascades, point
        # lights and distance LODs, at an odd size.
        _frame(name="frame_bounce_sky_541p", scene="room", triangles=60001, width=961, height=541, rays=4, samples=8,
               bounce=True, sky=True, lights=3, lod=True),
        # The dense layout: every probe of every level traces every direction.
        {"name": "dense_cornell", "kind": "dense", "probes": 64, "levels": 4},
        # Many views of many scenes per step through the batched entry point.
        {"name": "batch_12views", "kind": "batch", "views": 12, "rays": 36, "levels": 8, "scale": 2},
        # The learned-cache form of the benchmark frame: far cascades answered
        # by the MLP, which trains inside the frame.
        {"name": "learned_720p", "kind": "learned", "triangles": 262144, "width": 1280, "height": 720, "rays": 36,
         "cutoff": 1},
        # Caller rays: closest hits and occlusion over interval-sized limits.
        {"name": "trace_rays_300k", "kind": "trace", "triangles": 20000, "rays": 300007},
        # Radiance of a few caller rays (light probes, picking).
        {"name": "radiance_rays_4k", "kind": "radiance", "triangles": 20000, "rays": 4099, "samples": 16},
        # Screen reconstruction after the resolve: temporal and three passes.
        {"name": "screen_720p", "kind": "screen", "width": 1280, "height": 720, "passes": 3},
        # The learned cache by itself: one frame's training and its queries.
        {"name": "cache_train_query", "kind": "cache", "train": 65536, "queries": 500009},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "dense", "batch", "learned", "trace", "radiance", "screen",
                       "cache"])
    if kind == "frame":
        width = _log(rng, 48, 1600)
        height = max(27, int(width * rng.uniform(0.5, 0.75)))
        levels = rng.randint(3, 8)
        stride = rng.choice([2, 3, 4, 4, 4])
        most = max(1, 2_000_000 // max(1, (width // stride) * (height // stride)))
        bounce = levels <= 4 and rng.random() < 0.4
        sky = rng.random() < 0.3
        return _frame(scene="room", triangles=_log(rng, 1000, 200000), width=width, height=height, stride=stride,
                      points=rng.choice([1, 1, 2]), rays=min(rng.choice([1, 1, 2, 4, 9, 16, 36]), most), levels=levels,
                      ratio=4.0 if levels <= 4 else 2.0, samples=rng.choice([4, 8, 16] if sky else [4, 16, 16, 24]),
                      history=rng.random() < 0.8, host=rng.random() < 0.3, sort=rng.random() < 0.4, bounce=bounce,
                      sky=sky, lights=rng.choice([0, 0, 1, 3]) if not sky else 0,
                      lod=levels <= 4 and rng.random() < 0.3)
    if kind == "dense":
        return {"kind": "dense", "probes": rng.randint(9, 96), "levels": rng.randint(2, 4)}
    if kind == "batch":
        return {"kind": "batch", "views": rng.randint(2, 12), "rays": rng.choice([1, 4, 16, 36]),
                "levels": rng.randint(4, 8), "scale": rng.choice([2, 3, 4])}
    if kind == "learned":
        width = _log(rng, 320, 1280)
        return {"kind": "learned", "triangles": 2 * _log(rng, 104000, 200000), "width": width,
                "height": int(width * 0.5625), "rays": rng.choice([9, 16, 36]), "cutoff": rng.choice([1, 2, 3])}
    if kind == "trace":
        return {"kind": "trace", "triangles": _log(rng, 1000, 40000), "rays": _log(rng, 100, 400000)}
    if kind == "radiance":
        return {"kind": "radiance", "triangles": _log(rng, 1000, 200000), "rays": _log(rng, 100, 600000),
                "samples": rng.choice([4, 8, 16, 32])}
    if kind == "screen":
        width = _log(rng, 160, 1920)
        return {"kind": "screen", "width": width, "height": max(90, int(width * rng.uniform(0.5, 0.7))),
                "passes": rng.randint(0, 4)}
    return {"kind": "cache", "train": _log(rng, 1000, 131072), "queries": _log(rng, 1000, 1500000)}


# ---- scenes and cameras ------------------------------------------------------


@functools.lru_cache(maxsize=24)
def _packed(scene, triangles):
    """(description, packed words, emitter instances) of a scene; geometry
    depends on the case alone."""
    emitters = []
    if scene == "cornell":
        desc = scenes.cornell()
    elif scene == "atrium":
        desc = scenes.atrium(seed=2, triangles=triangles)
    elif scene == "full":
        desc, emitters, _ = scenes.full_scene(5, triangles)
    else:
        desc = scenes.batch_scene(3000 + triangles, triangles)
    return desc, bp.PackedScene.from_desc(desc), emitters


def _camera(scene, triangles, rng):
    """Eye and target of a view into the scene, moved a little by the seed."""
    if scene == "cornell":
        eye, target, move = (0.0, 1.0, 3.1), (0.0, 0.9, 0.0), 0.1
    elif scene in ("atrium", "full"):
        if triangles >= 200_000:
            eye, target, move = (-17.0, 3.0, -15.0), (4.0, 4.0, 6.0), 0.5
        else:
            eye, target, move = (-7.0, 3.0, -6.5), (2.0, 3.0, 3.0), 0.3
    else:
        size = 6.0 + 18.0 * math.log(triangles / 1000.0 + 1.0) / math.log(201.0)
        height = 3.0 + 0.25 * size
        eye, target = (0.05 * size, 0.45 * height, -0.45 * size), (-0.05 * size, 0.2 * height, 0.3 * size)
        move = 0.02 * size
    return (tuple(float(v) for v in np.asarray(eye) + rng.uniform(-move, move, 3)),
            tuple(float(v) for v in np.asarray(target) + rng.uniform(-move, move, 3)))


@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream(DEVICE)


def _context():
    return bp.LuxContext(0, _stream().cuda_stream)


def _primary(ctx, scene, packed, eye, target, width, height, stride):
    """First surfaces of the camera's pixel blocks: position, normal facing
    the camera, view depth, instance, and the blocks that hit."""
    def unit(v):
        return v / np.linalg.norm(v)
    fwd = unit(np.asarray(target, np.float64) - np.asarray(eye, np.float64))
    right = unit(np.cross(fwd, (0.0, 1.0, 0.0)))
    up = np.cross(right, fwd)
    tan = math.tan(math.radians(FOV) * 0.5)
    f64 = dict(dtype=torch.float64, device=DEVICE)
    xs = (torch.arange(0, width, stride, **f64) + stride * 0.5) / width * 2.0 - 1.0
    ys = 1.0 - (torch.arange(0, height, stride, **f64) + stride * 0.5) / height * 2.0
    gy, gx = torch.meshgrid(ys, xs, indexing="ij")
    d = (torch.tensor(fwd, **f64) + gx[..., None] * (tan * width / height) * torch.tensor(right, **f64)
         + gy[..., None] * tan * torch.tensor(up, **f64)).reshape(-1, 3)
    d = (d / d.norm(dim=1, keepdim=True)).float()
    rays = torch.zeros((len(d), 8), device=DEVICE)
    rays[:, 0:3] = torch.tensor(eye, device=DEVICE)
    rays[:, 4:7] = d
    rays[:, 7] = 1e20
    hits = torch.zeros((len(d), 8), dtype=torch.int32, device=DEVICE)
    torch.cuda.synchronize()
    bp.trace_rays(ctx, scene, rays.data_ptr(), len(d), hits.data_ptr())
    index = torch.nonzero(hits[:, 1] != EMPTY).reshape(-1)
    d, hits = d[index], hits[index]
    t = hits.view(torch.float32)[:, 0:1]
    pos = torch.zeros((len(d), 4), device=DEVICE)
    pos[:, :3] = rays[0, 0:3] + d * t
    # World normals of the hit triangles from the packed words.
    sw = torch.from_numpy(packed.scene_words.view(np.int32)).to(DEVICE)
    gw = torch.from_numpy(packed.geometry_words.view(np.int32)).to(DEVICE)
    header = packed.scene_words[0].astype(np.int64)
    vertices = int(packed.geometry_words[0][1])
    base = int(header[1]) + hits[:, 2].long() * int(header[3])
    corner = gw[1 + hits[:, 1].long()][:, :3].long()
    local = gw[vertices + corner * 5].view(torch.float32)[:, :, :3].double()
    rows = torch.stack([sw[base + 3 + r] for r in range(3)], 1).view(torch.float32).double()
    world = torch.einsum("nrc,nvc->nvr", rows[:, :, :3], local)
    n = torch.linalg.cross(world[:, 1] - world[:, 0], world[:, 2] - world[:, 0])
    n = n / n.norm(dim=1, keepdim=True).clamp_min(1e-30)
    n = torch.where(((n * d).sum(1, keepdim=True) > 0), -n, n).float()
    nrm = torch.zeros_like(pos)
    nrm[:, :3] = n
    depth = (t[:, 0].double() * (d.double() @ torch.tensor(fwd, **f64))).float()
    return pos, nrm, depth, hits[:, 2].contiguous(), index


def _image(pos, nrm, index, count):
    """Positions and normals of every pixel block; background blocks have a
    zero normal, which the resolve leaves unsupported."""
    full = [torch.zeros((count, 4), device=DEVICE) for _ in range(2)]
    full[0][index], full[1][index] = pos, nrm
    return full


def _blocks(width, height, stride):
    return -(-width // stride) * -(-height // stride)


def _settings(levels, ratio, rays=1, **fields):
    return bp.RadianceCascades(probe_spacing=0.25, interval_length=0.4, levels=levels, base_columns=8, base_rows=4,
                               interval_ratio=ratio, rays_per_receiver=rays, **fields).sanitized()


def _capacities(settings, pos, slack=1.0):
    """Cells (most of any level) and records (all levels) that receivers at
    `pos` seed."""
    cells, entries = 1, 1
    for level in range(settings.levels):
        grid = torch.floor(pos[:, :3] / (settings.probe_spacing * (1 << level))).long() + (1 << 18)
        keys = (grid[:, 0] << 40) | (grid[:, 1] << 20) | grid[:, 2]
        count = int(torch.unique(keys).numel())
        cells = max(cells, count)
        entries += count * ((8 << level) * (4 << level))
    return int(cells * slack) + 1, int(entries * slack) + 1


# ---- frames --------------------------------------------------------------------


def _prepare_frame(case, seed):
    rng = np.random.default_rng(seed)
    desc, packed, emitters = _packed(case["scene"], case["triangles"])
    eye, target = _camera(case["scene"], case["triangles"], rng)
    if case["lights"]:
        lights = []
        for _ in range(case["lights"]):
            at = np.asarray(eye) + (np.asarray(target) - eye) * rng.uniform(0.2, 0.9) + rng.uniform(-0.4, 0.4, 3)
            lights.append(bp.conventional_light(at, 8.0, rng.uniform(1.0, 6.0, 3)))
        packed = packed.with_conventional_lights(lights)
    ctx = _context()
    scene = bp.GpuScene(ctx, packed)
    fields = {"emissive_samples": case["samples"], "frame_index": int(rng.integers(0, 4096)),
              "history_frames": 24 if case["history"] else 0}
    if case["sky"]:
        fields["environment"] = (0.3, 0.4, 0.6)
    if case["bounce"]:
        fields.update(multi_bounce=True, cached_hit_sky=case["sky"])
    settings = _settings(case["levels"], case["ratio"], case["rays"], **fields)
    rpos, rnrm, _, _, _ = _primary(ctx, scene, packed, eye, target, case["width"], case["height"], case["stride"])
    ppos, pnrm, _, _, index = _primary(ctx, scene, packed, eye, target, case["width"], case["height"], case["points"])
    ppos, pnrm = _image(ppos, pnrm, index, _blocks(case["width"], case["height"], case["points"]))
    cells, entries = _capacities(settings, rpos, 2.0 if case["lod"] else 1.0)
    if case["bounce"]:  # the secondary cascades' receivers spread over the whole scene
        cells, entries = max(cells, len(rpos)), 3 * entries + (1 << 20)
    view = bp.SplitView(ctx, max_receivers=len(rpos), max_cells=cells, max_entries=entries,
                        max_rays=len(rpos) * case["rays"])
    if case["sort"]:
        view.set_tuning(sort_queries=1, stack_depth=32, closest_blocks_per_sm=8, shadow_blocks_per_sm=8)
    if case["lod"]:
        view.set_camera(scenes.clip_from_world(eye, target, FOV, case["width"], case["height"]), eye, case["height"], 8)
    state = dict(kind="frame", ctx=ctx, scene=scene, view=view, settings=settings, frame=0, moves=None,
                 host=case["host"], packed=packed)
    if case["host"]:
        arrays = [t.cpu().pin_memory() for t in (rpos, rnrm, ppos, pnrm)]
        out = torch.zeros((len(ppos), 4)).pin_memory()
        state.update(buffers=arrays, arrays=[a.numpy() for a in arrays], out=out, out_array=out.numpy())
    else:
        state.update(rpos=rpos, rnrm=rnrm, ppos=ppos, pnrm=pnrm, out=torch.zeros((len(ppos), 4), device=DEVICE))
    if case["moving"]:
        state["moves"] = _emitter_moves(desc, packed, emitters, rng)
    torch.cuda.synchronize()
    run(state)  # the view's second frame on: history, sort buffers and the secondary cascades exist
    if view.stats().error_flags:
        raise RuntimeError("the view's capacities do not hold the case")
    return state


def _emitter_moves(desc, packed, emitters, rng):
    """Slot-ordered poses of eight successive frames and the boxes around the
    emitters that moved."""
    order = packed.instance_order.astype(np.int64)
    slot = np.empty(len(order), np.int64)
    slot[order] = np.arange(len(order))
    base = np.stack([desc.instance_transform[int(i)] for i in order]).astype(np.float64)
    start = float(rng.uniform(0.0, 10.0))
    moves = []
    for frame in range(8):
        poses, boxes = base.copy(), []
        for centre, radius, phase, sign in scenes.emitter_orbits(desc, emitters):
            angle = phase + sign * 0.5 * (start + frame / 60.0) / radius
            at = centre + radius * np.array([math.cos(angle), 0.0, math.sin(angle)])
            k = len(boxes)
            poses[slot[emitters[k]], :, 3] = at
            boxes.append((at - (1.1, 0.1, 1.1), at + (1.1, 0.1, 1.1)))
        moves.append((poses.astype(np.float32), boxes))
    return moves


def _run_frame(s):
    view, scene, settings = s["view"], s["scene"], s["settings"]
    settings.frame_index += 1
    s["frame"] += 1
    if s["moves"] is not None:
        poses, boxes = s["moves"][s["frame"] % len(s["moves"])]
        scene.refit(poses, s["packed"].lights_at(poses))
        for lo, hi in boxes:
            view.invalidate_bounds(lo, hi)
    if s["host"]:
        rpos, rnrm, ppos, pnrm = s["arrays"]
        view.frame_host(scene, settings, rpos, rnrm, ppos, pnrm, out=s["out_array"])
        return s["out"]
    view.trace_merge(scene, settings, s["rpos"].data_ptr(), s["rnrm"].data_ptr(), len(s["rpos"]))
    view.resolve(settings, s["ppos"].data_ptr(), s["pnrm"].data_ptr(), len(s["ppos"]), s["out"].data_ptr())
    return s["out"]


def _prepare_dense(case, seed):
    rng = np.random.default_rng(seed)
    _, packed, _ = _packed("cornell", 34)
    ctx = _context()
    scene = bp.GpuScene(ctx, packed)
    settings = bp.RadianceCascades(probe_spacing=0.1, interval_length=0.05, levels=case["levels"], base_columns=4,
                                   base_rows=4, interval_ratio=2.0, layout=bp.LAYOUT_DENSE,
                                   interval_rule=bp.INTERVAL_LENGTHS_GEOMETRIC,
                                   frame_index=int(rng.integers(0, 4096))).sanitized()
    pos, nrm = scenes.dense_plane_probes(case["probes"], 0.1, int(rng.integers(2, 18)))
    pos, nrm = torch.from_numpy(pos).to(DEVICE), torch.from_numpy(nrm).to(DEVICE)
    cells, entries, records = 1, 1, 0
    for level in range(settings.levels):
        grid = torch.floor(pos[:, :3] / (0.1 * (1 << level)) + 1e-3).long()
        count = int(torch.unique(grid, dim=0).shape[0]) + 8
        cells, entries = max(cells, 2 * count), entries + 2 * count * (16 << (2 * level))
        records += 2 * count * (16 << (2 * level))
    view = bp.SplitView(ctx, max_receivers=len(pos), max_cells=cells, max_entries=entries, max_rays=records)
    eye, target = _camera("cornell", 34, rng)
    ppos, pnrm, _, _, index = _primary(ctx, scene, packed, eye, target, DENSE_WIDTH, DENSE_HEIGHT, 1)
    ppos, pnrm = _image(ppos, pnrm, index, DENSE_WIDTH * DENSE_HEIGHT)
    state = dict(kind="frame", ctx=ctx, scene=scene, view=view, settings=settings, frame=0, moves=None, host=False,
                 packed=packed, rpos=pos, rnrm=nrm, ppos=ppos, pnrm=pnrm,
                 out=torch.zeros((len(ppos), 4), device=DEVICE))
    torch.cuda.synchronize()
    run(state)
    if view.stats().error_flags:
        raise RuntimeError("the view's capacities do not hold the case")
    return state


def _batch_jobs(case):
    """(triangles, width, height) of the batch's views: the batched
    workload's first scenes, their resolutions divided by `scale`."""
    return [(2 * (triangles // 2), width // case["scale"], height // case["scale"])
            for _, triangles, (width, height) in scenes.batch_workload(seed=3, scenes=case["views"])]


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    ctx = _context()
    settings = _settings(case["levels"], 2.0, case["rays"], emissive_samples=16,
                         frame_index=int(rng.integers(0, 4096)))
    jobs, keep, outs = [], [], []
    for triangles, width, height in _batch_jobs(case):
        _, packed, _ = _packed("room", triangles)
        scene = bp.GpuScene(ctx, packed)
        eye, target = _camera("room", triangles, rng)
        pos, nrm, _, _, index = _primary(ctx, scene, packed, eye, target, width, height, 4)
        points = _image(pos, nrm, index, _blocks(width, height, 4))
        cells, entries = _capacities(settings, pos)
        view = bp.SplitView(ctx, max_receivers=len(pos), max_cells=cells, max_entries=entries,
                            max_rays=len(pos) * case["rays"])
        jobs.append((view, scene, pos.data_ptr(), nrm.data_ptr(), len(pos)))
        keep.append((pos, nrm, *points))
        outs.append(torch.zeros((len(points[0]), 4), device=DEVICE))
    batch = bp.Batch(ctx)
    state = dict(kind="batch", ctx=ctx, batch=batch, jobs=jobs, keep=keep, outs=outs, settings=settings)
    torch.cuda.synchronize()
    run(state)  # the frame is captured once and replayed from then on
    run(state)
    for view, *_ in jobs:
        if view.stats().error_flags:
            raise RuntimeError("a view's capacities do not hold the case")
    return state


def _run_batch(s):
    settings = s["settings"]
    settings.frame_index += 1
    s["batch"].trace_merge(s["jobs"], settings)
    for (view, *_), (_, _, ppos, pnrm), out in zip(s["jobs"], s["keep"], s["outs"]):
        view.resolve(settings, ppos.data_ptr(), pnrm.data_ptr(), len(ppos), out.data_ptr())
    return s["outs"]


def _prepare_learned(case, seed):
    rng = np.random.default_rng(seed)
    _, packed, _ = _packed("atrium", case["triangles"])
    ctx = _context()
    scene = bp.GpuScene(ctx, packed)
    eye, target = _camera("atrium", case["triangles"], rng)
    settings = _settings(8, 2.0, case["rays"], emissive_samples=16, frame_index=int(rng.integers(0, 4096)))
    rpos, rnrm, _, _, _ = _primary(ctx, scene, packed, eye, target, case["width"], case["height"], 4)
    ppos, pnrm, _, _, index = _primary(ctx, scene, packed, eye, target, case["width"], case["height"], 1)
    ppos, pnrm = _image(ppos, pnrm, index, case["width"] * case["height"])
    cells, entries = _capacities(settings, rpos)
    view = bp.SplitView(ctx, max_receivers=len(rpos), max_cells=cells, max_entries=entries,
                        max_rays=len(rpos) * case["rays"])
    cache = bp.LearnedCache(ctx, seed=int(rng.integers(1, 1 << 20)))
    cache.set_bounds((rpos[:, :3].min(0).values - 1.0).cpu().numpy(), (rpos[:, :3].max(0).values + 1.0).cpu().numpy())
    view.set_cache(cache, cutoff_level=case["cutoff"], validate_period=16, error_bound=8.0, train_samples=65536,
                   fallback_frames=16)
    state = dict(kind="frame", ctx=ctx, scene=scene, view=view, settings=settings, frame=0, moves=None, host=False,
                 packed=packed, cache=cache, rpos=rpos, rnrm=rnrm, ppos=ppos, pnrm=pnrm,
                 out=torch.zeros((len(ppos), 4), device=DEVICE))
    torch.cuda.synchronize()
    for _ in range(4):
        run(state)
    if view.stats().error_flags or cache.stats().error_flags:
        raise RuntimeError("the learned-cache frame reports an error")
    return state


# ---- caller rays ---------------------------------------------------------------


def _interval_rays(case, seed):
    """Rays of the room scene as float32[n, 8] (origin, tmin, direction,
    limit): origins in the room's free space, directions over the sphere,
    limits from the cascades' interval ends and the room's length."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    n = case["rays"]
    size = 6.0 + 18.0 * math.log(case["triangles"] / 1000.0 + 1.0) / math.log(201.0)
    height = 3.0 + 0.25 * size
    rays = torch.zeros((n, 8), device=DEVICE)
    span = torch.tensor([0.94 * size, 0.9 * height, 0.94 * size], device=DEVICE)
    low = torch.tensor([-0.47 * size, 0.05 * height, -0.47 * size], device=DEVICE)
    rays[:, 0:3] = low + span * torch.rand((n, 3), generator=g, device=DEVICE)
    d = torch.randn((n, 3), generator=g, device=DEVICE)
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    ends = torch.tensor([0.4, 1.6, 6.4, 25.6, 2.0 * size], device=DEVICE)
    starts = torch.tensor([0.0, 0.4, 1.6, 0.0, 0.0], device=DEVICE)
    level = torch.randint(0, 5, (n,), generator=g, device=DEVICE)
    rays[:, 3], rays[:, 7] = starts[level], ends[level]
    return rays


def _prepare_trace(case, seed):
    _, packed, _ = _packed("room", case["triangles"])
    ctx = _context()
    scene = bp.GpuScene(ctx, packed)
    rays = _interval_rays(case, seed)
    hits = [torch.zeros((len(rays), 8), dtype=torch.int32, device=DEVICE) for _ in range(2)]
    torch.cuda.synchronize()
    return dict(kind="trace", ctx=ctx, scene=scene, rays=rays, hits=hits)


def _run_trace(s):
    rays, (near, any_) = s["rays"], s["hits"]
    bp.trace_rays(s["ctx"], s["scene"], rays.data_ptr(), len(rays), near.data_ptr())
    bp.trace_rays(s["ctx"], s["scene"], rays.data_ptr(), len(rays), any_.data_ptr(), any_hit=True)
    values = near.view(torch.float32)
    with torch.cuda.stream(_stream()):
        blocked = any_[:, 1] != EMPTY
    return {"distance": values[:, 0], "barycentric": values[:, 4:7], "triangle": near[:, 1], "instance": near[:, 2],
            "errors": near[:, 3], "blocked": blocked}


def _prepare_radiance(case, seed):
    _, packed, _ = _packed("room", case["triangles"])
    ctx = _context()
    scene = bp.GpuScene(ctx, packed)
    rays = _interval_rays(case, seed)
    rays[:, 3], rays[:, 7] = 0.0, 1e20
    settings = _settings(4, 4.0, emissive_samples=case["samples"], frame_index=seed % 4096)
    out = torch.zeros((len(rays), 4), device=DEVICE)
    torch.cuda.synchronize()
    return dict(kind="radiance", ctx=ctx, scene=scene, rays=rays, settings=settings, out=out)


def _run_radiance(s):
    rays = s["rays"]
    bp.interval_radiance(s["ctx"], s["scene"], s["settings"], rays.data_ptr(), len(rays), s["out"].data_ptr())
    # An escaped ray's distance is its limit (1e20): radiance and distance apart.
    return {"radiance": s["out"][:, :3], "distance": s["out"][:, 3].clamp(max=1e4)}


# ---- screen reconstruction -----------------------------------------------------


def _screen_frames(case, seed):
    """Two successive frames (irradiance, position, normal, identity,
    clip_from_world) of a camera that moves a little."""
    rng = np.random.default_rng(seed)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    _, packed, _ = _packed("atrium", 65536)
    ctx = _context()
    scene = bp.GpuScene(ctx, packed)
    eye, target = _camera("atrium", 65536, rng)
    width, height = case["width"], case["height"]
    frames = []
    for k in range(2):
        at = (eye[0] + 0.02 * k, eye[1] + 0.005 * k, eye[2] + 0.015 * k)
        pos, nrm, depth, inst, index = _primary(ctx, scene, packed, at, target, width, height, 1)
        n = width * height
        position, normal = torch.zeros((n, 4), device=DEVICE), torch.zeros((n, 4), device=DEVICE)
        irradiance, identity = torch.zeros((n, 4), device=DEVICE), torch.zeros((n, 2), dtype=torch.int32, device=DEVICE)
        position[index] = torch.cat([pos[:, :3], depth[:, None]], 1)
        normal[index] = nrm
        identity[index, 0] = inst
        base = 0.4 + 0.3 * torch.sin(pos[:, :3] * torch.tensor([0.7, 1.1, 0.9], device=DEVICE))
        value = base * torch.exp(0.5 * torch.randn((len(pos), 3), generator=g, device=DEVICE))
        u = torch.rand((len(pos), 1), generator=g, device=DEVICE)
        cover = torch.where(u < 0.7, torch.ones_like(u), u)
        alpha = torch.where(u < 0.05, torch.full_like(u, -1.0), 1.0 + 0.25 * cover)
        irradiance[index] = torch.cat([value, alpha], 1)
        frames.append((irradiance, position, normal, identity,
                       scenes.clip_from_world(at, target, FOV, width, height)))
    torch.cuda.synchronize()
    return ctx, scene, frames


def _prepare_screen(case, seed):
    ctx, scene, frames = _screen_frames(case, seed)
    settings = _settings(4, 4.0)
    screen = bp.ScreenFilter(ctx, case["width"], case["height"])
    out = torch.zeros((case["height"], case["width"], 4), device=DEVICE)
    torch.cuda.synchronize()
    state = dict(kind="screen", ctx=ctx, scene=scene, frames=frames, settings=settings, screen=screen, out=out, frame=0,
                 passes=case["passes"])
    run(state)
    return state


def _run_screen(s):
    irradiance, position, normal, identity, _ = s["frames"][s["frame"] % 2]
    previous = s["frames"][(s["frame"] + 1) % 2][4]
    s["frame"] += 1
    s["screen"].filter(s["settings"], irradiance.data_ptr(), position.data_ptr(), normal.data_ptr(),
                       identity.data_ptr(), previous, s["out"].data_ptr(), spatial_filter_steps=s["passes"])
    return s["out"]


# ---- learned cache -------------------------------------------------------------


def _cache_samples(n, g):
    """Device records (float32[n, 16]) of points in a 40 x 10 x 40 m hall."""
    s = torch.zeros((n, 16), device=DEVICE)
    s[:, 0:3] = torch.rand((n, 3), generator=g, device=DEVICE) * torch.tensor([40.0, 10.0, 40.0], device=DEVICE)
    s[:, 3] = 1.0
    for at in (4, 8):
        v = torch.randn((n, 3), generator=g, device=DEVICE)
        s[:, at:at + 3] = v / v.norm(dim=1, keepdim=True)
    return s


def _prepare_cache(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    ctx = _context()
    cache = bp.LearnedCache(ctx, seed=1 + seed % 65536)
    cache.set_bounds((0.0, 0.0, 0.0), (40.0, 10.0, 40.0))
    samples, queries = _cache_samples(case["train"], g), _cache_samples(case["queries"], g)
    target = torch.zeros((case["train"], 4), device=DEVICE)
    wave = torch.sin(samples[:, 0:3] * torch.tensor([0.21, 0.5, 0.17], device=DEVICE))
    target[:, :3] = (1.0 + wave) * torch.exp(0.4 * torch.randn((case["train"], 3), generator=g, device=DEVICE))
    out = torch.zeros((case["queries"], 4), device=DEVICE)
    torch.cuda.synchronize()
    return dict(kind="cache", ctx=ctx, cache=cache, samples=samples, target=target, queries=queries, out=out)


def _run_cache(s):
    cache = s["cache"]
    cache.train(s["samples"].data_ptr(), s["target"].data_ptr(), len(s["samples"]))
    cache.query(s["queries"].data_ptr(), len(s["queries"]), s["out"].data_ptr())
    return {"radiance": s["out"], "weights": cache.weights()}


# ---- the interface ---------------------------------------------------------------

_PREPARE = {"frame": _prepare_frame, "dense": _prepare_dense, "batch": _prepare_batch, "learned": _prepare_learned,
            "trace": _prepare_trace, "radiance": _prepare_radiance, "screen": _prepare_screen,
            "cache": _prepare_cache}
_RUN = {"frame": _run_frame, "batch": _run_batch, "trace": _run_trace, "radiance": _run_radiance,
        "screen": _run_screen, "cache": _run_cache}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


# Operations of a walk that nothing shorter answers: the tests along one path
# of the tree (log4 of the triangles, four boxes of 20 operations each) and
# two triangles of 60.
def _walk(triangles):
    return 80.0 * math.log(max(triangles, 4), 4) + 120.0


def _frame_work(receivers, points, rays, levels, samples, triangles, scene_bytes, history=True, directions=32):
    """One Split frame: receivers and points read, the scene read, irradiance
    written; a closest-hit walk per ray, a visibility walk per next-event
    sample of the rays that hit; one deposit per ray; the records the rays
    reached read, blended and merged (60 bytes, 84 with history)."""
    traced = receivers * rays
    records = min(traced * levels, 20_000_000)
    flops = traced * _walk(triangles) + 0.6 * traced * max(1, samples // 2) * (_walk(triangles) + 60.0)
    flops += records * 40.0 + points * 200.0
    return {"bytes": 32.0 * receivers + 48.0 * points + scene_bytes + records * (84.0 if history else 60.0),
            "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "frame":
        receivers = (case["width"] // case["stride"]) * (case["height"] // case["stride"])
        points = (case["width"] // case["points"]) * (case["height"] // case["points"])
        w = _frame_work(receivers, points, case["rays"], case["levels"], case["samples"], case["triangles"],
                        100.0 * case["triangles"], case["history"])
        return {k: v * (2.0 if case["bounce"] else 1.0) for k, v in w.items()}
    if kind == "dense":
        cells, rays = case["probes"] ** 2, 0
        for level in range(case["levels"]):
            rays += (cells >> (2 * level)) * (16 << (2 * level))
        return {"bytes": 60.0 * rays + 16.0 * cells + 48.0 * DENSE_WIDTH * DENSE_HEIGHT,
                "flops": rays * (_walk(34) + 0.6 * 8 * (_walk(34) + 60.0) + 40.0)}
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for triangles, width, height in _batch_jobs(case):
            receivers = (width // 4) * (height // 4)
            w = _frame_work(receivers, receivers, case["rays"], case["levels"], 16, triangles, 100.0 * triangles)
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "learned":
        receivers, points = (case["width"] // 4) * (case["height"] // 4), case["width"] * case["height"]
        w = _frame_work(receivers, points, case["rays"], case["cutoff"] + 1, 4, case["triangles"],
                        100.0 * case["triangles"])
        network = 2.0 * (4 * 64 * 64 + 16 * 64)
        w["flops"] += receivers * case["rays"] * 0.8 * network + 65536 * 3.0 * network
        w["bytes"] += receivers * case["rays"] * 0.8 * 16.0 + 65536 * 80.0
        return w
    if kind == "trace":
        return {"bytes": 2.0 * 64.0 * case["rays"] + 100.0 * case["triangles"],
                "flops": 2.0 * case["rays"] * _walk(case["triangles"])}
    if kind == "radiance":
        walk = _walk(case["triangles"])
        return {"bytes": 48.0 * case["rays"] + 100.0 * case["triangles"],
                "flops": case["rays"] * (walk + max(1, case["samples"] // 2) * (walk + 60.0))}
    if kind == "screen":
        n = case["width"] * case["height"]
        # Inputs and history read, history and output written, once each.
        return {"bytes": n * (56.0 + 72.0 + 72.0 + 16.0), "flops": n * (400.0 + 21.0 * 60.0 * case["passes"])}
    network = 2.0 * (4 * 64 * 64 + 16 * 64)
    touched = min(case["train"] * 8.0, float(1 << 19)) * 16
    return {"bytes": case["train"] * 80.0 + case["queries"] * 80.0 + touched * 28.0,
            "flops": case["train"] * 3.0 * network + case["queries"] * network}


# ---- 64-bit values -------------------------------------------------------------


def exact(case, seed):
    """Closest distances by testing every ray against every triangle, and the
    screen filter by its formulas; the other outputs rest on integer sample
    sequences, BF16 training or float atomics and have no short definition."""
    if case["kind"] == "trace":
        return _exact_trace(case, seed)
    if case["kind"] == "screen":
        return _exact_screen(case, seed)
    return None


def _exact_trace(case, seed):
    desc, _, _ = _packed("room", case["triangles"])
    rays = _interval_rays(case, seed).double()
    world = []
    for mesh, m in zip(desc.instance_mesh, desc.instance_transform):
        m = np.asarray(m, np.float32).astype(np.float64)
        v = np.asarray(desc.meshes[mesh].positions, np.float32).astype(np.float64) @ m[:, :3].T + m[:, 3]
        world.append(v[desc.meshes[mesh].indices])
    tri = torch.from_numpy(np.concatenate(world)).to(DEVICE)
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    best = rays[:, 7].clone()
    chunk = max(1, 24_000_000 // len(tri))
    for first in range(0, len(rays), chunk):
        r = rays[first:first + chunk]
        o, d = r[:, 0:3], r[:, 4:7]
        det = -(d @ n.T)
        # Moeller-Trumbore by triple products: d x (o - a) expanded per ray.
        od = torch.linalg.cross(o, d)  # o x d
        t = (o @ n.T - (a * n).sum(1)) / det
        c1 = (od @ e2.T) - d @ torch.linalg.cross(e2, a).T
        u = c1 / det
        c2 = (od @ e1.T) - d @ torch.linalg.cross(e1, a).T
        v = -c2 / det
        low = torch.clamp(r[:, 3:4], min=2.5e-5)
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > low) & (t < r[:, 7:8])
        t = torch.where(ok, t, torch.full_like(t, math.inf)).min(1).values
        best[first:first + chunk] = torch.minimum(best[first:first + chunk], t)
    return {"distance": best, "barycentric": None, "triangle": None, "instance": None, "errors": None, "blocked": None}


def _shift(image, dy, dx, fill=0.0):
    """image[y + dy, x + dx], `fill` outside."""
    h, w = image.shape[:2]
    out = torch.full_like(image, fill)
    y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
    if y0 < y1 and x0 < x1:
        out[y0:y1, x0:x1] = image[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
    return out


def _luminance(c):
    return c[..., 0] * 0.2126 + c[..., 1] * 0.7152 + c[..., 2] * 0.0722


def _plane(delta, target, sample):
    mean = target + sample
    length = mean.norm(dim=-1, keepdim=True)
    n = torch.where(length > 1e-10, mean / length.clamp_min(1e-30), target)
    return (delta * n).sum(-1).abs()


def _exact_screen(case, seed):
    h, w = case["height"], case["width"]
    _, _, frames = _screen_frames(case, seed)
    tolerance, scale = max(0.005 * 2.0, 0.25 * 0.02), max(0.005 * 2.0, 0.25 * 0.05)
    blend, capacity = float(np.float32(0.88)), 24.0
    history = None
    images = []
    for irr, pos, nrm, ident, clip in frames:
        images.append((irr.double().view(h, w, 4), pos.double().view(h, w, 4), nrm.double().view(h, w, 4)[..., :3],
                       ident.view(h, w, 2)[..., 0].long(), torch.from_numpy(clip).double().to(DEVICE)))
    for k, (irr, pos, nrm, ident, _) in enumerate(images):
        previous = images[1 - k][4]
        surface = pos[..., 3] > 0
        mask = (irr[..., 3] > 0) & ((torch.floor(irr[..., 3]).long() & 1) == 1)
        supported = mask & surface
        fresh = torch.where(supported, ((irr[..., 3] - torch.floor(irr[..., 3])) * 4.0).clamp(0, 1), 0.0)
        center = torch.where(supported[..., None], irr[..., :3], 0.0)
        total = torch.zeros((h, w, 3), dtype=torch.float64, device=DEVICE)
        square, count = torch.zeros_like(total), torch.zeros((h, w), dtype=torch.float64, device=DEVICE)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                v, op, on = _shift(irr, dy, dx), _shift(pos, dy, dx), _shift(nrm, dy, dx)
                omask = (torch.floor(v[..., 3]).long() & 1) == 1
                ok = (v[..., 3] > 0) & (~mask | omask) & (op[..., 3] > 0) & (_shift(ident, dy, dx, -1) == ident)
                ok &= ((nrm * on).sum(-1) > 0.97) & (_plane(op[..., :3] - pos[..., :3], nrm, on) <= tolerance)
                weight = ok.double()[..., None]
                total, square = total + v[..., :3] * weight, square + v[..., :3] ** 2 * weight
                count = count + weight[..., 0]
        div = count.clamp_min(1.0)[..., None]
        mean = total / div
        var = (square / div - mean * mean).clamp_min(0.0)
        dev = var.sqrt()
        retained = fresh.clone()
        variance = torch.where(supported, _luminance(var), 0.0)
        if history is not None:
            hirr, hmeta, hpos, hnrm, hid = history
            c = pos[..., :3] @ previous[:, :3].T + previous[:, 3]
            px, py = (c[..., 0] / c[..., 3] * 0.5 + 0.5) * w, (0.5 - c[..., 1] / c[..., 3] * 0.5) * h
            inside = (c[..., 3] > 0) & (px >= 0) & (py >= 0) & (px < w) & (py < h) & surface
            lx, ly = torch.where(inside, px, 0.5) - 0.5, torch.where(inside, py, 0.5) - 0.5
            bx, by = torch.floor(lx).long(), torch.floor(ly).long()
            left, top = bx.clamp(max=w - 1), by.clamp(max=h - 1)
            fx = ((lx - left) / ((bx + 1).clamp(max=w - 1) - left).clamp_min(1)).clamp(0, 1)
            fy = ((ly - top) / ((by + 1).clamp(max=h - 1) - top).clamp_min(1)).clamp(0, 1)
            old, om, weights = torch.zeros_like(total), torch.zeros_like(total)[..., :2], torch.zeros_like(count)
            for corner in range(4):
                ox, oy = bx + (corner & 1), by + (corner >> 1)
                ok = inside & (ox >= 0) & (oy >= 0) & (ox < w) & (oy < h)
                at = (oy.clamp(0, h - 1), ox.clamp(0, w - 1))
                v, m, p, n = hirr[at], hmeta[at], hpos[at], hnrm[at]
                ok &= (m[..., 0] > 0) & (v[..., 3] > 0) & (m[..., 3] > 0) & (hid[at] == ident) & (m[..., 2] > 0)
                ok &= ((nrm * n).sum(-1) > 0.97) & (_plane(p[..., :3] - pos[..., :3], nrm, n) <= tolerance)
                weight = (fx if corner & 1 else 1 - fx) * (fy if corner >> 1 else 1 - fy) * ok
                old, om = old + v[..., :3] * weight[..., None], om + m[..., :2] * weight[..., None]
                weights = weights + weight
            has = weights > 0.00001
            old, om = old / weights.clamp_min(1e-30)[..., None], om / weights.clamp_min(1e-30)[..., None]
            length = om[..., 0].clamp(max=capacity)
            complete = fresh >= 1.0
            d = _luminance(old) - _luminance(center)
            spread = 2.5 * torch.maximum(dev, torch.maximum(om[..., 1], d * d * 0.25).sqrt()[..., None]) + 0.0001
            clipped = torch.minimum(torch.maximum(old, (mean - spread).clamp_min(0.0)), mean + spread)
            clipped = torch.where((complete & (count >= 2))[..., None], clipped, old)
            weight = (length / (length + 1.0)).clamp(max=blend)
            weight = weight / (weight + fresh * (1 - weight)).clamp_min(1e-8)
            blended = center + weight[..., None] * (clipped - center)
            bvar = _luminance(var) + weight * (om[..., 1] - _luminance(var)) + weight * (1 - weight) * d * d
            use = has & supported & (fresh > 0.00001)
            keep = has & ~use
            center = torch.where(use[..., None], blended, torch.where(keep[..., None], old, center))
            retained = torch.where(use, (length + fresh).clamp(max=capacity), torch.where(keep, length, retained))
            variance = torch.where(use, bvar, torch.where(keep, om[..., 1], variance))
            mask = torch.where(has, torch.ones_like(mask), mask)
        depth = torch.where(supported | (retained > 0), pos[..., 3], 0.0)
        zero = ~surface
        image = torch.cat([center, depth[..., None]], -1)
        meta = torch.stack([retained, variance, mask.double(), torch.ones_like(variance)], -1)
        image[zero], meta[zero] = 0.0, 0.0
        history = (image, meta, torch.where(zero[..., None], 0.0, pos), torch.where(zero[..., None], 0.0, nrm),
                   torch.where(zero, 0, ident))
    image, meta, _, nrm, ident = history
    pos = images[1][1]
    mask = meta[..., 2] > 0
    kernel = (1.0, 4.0, 6.0, 4.0, 1.0)
    for level in range(case["passes"]):
        step = 1 << level
        light = image[..., 3] > 0
        depth = torch.where(light, image[..., 3], pos[..., 3])
        total, weights = torch.zeros_like(image[..., :3]), torch.zeros_like(depth)
        centre_l = _luminance(image)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                if abs(dy) == 2 and abs(dx) == 2:
                    continue
                v, om, on = (_shift(t, dy * step, dx * step) for t in (image, meta, nrm))
                ok = (v[..., 3] > 0) & (om[..., 0] > 0) & (om[..., 3] > 0) & (meta[..., 3] > 0)
                omask = _shift(mask.double(), dy * step, dx * step) > 0
                ok &= (_shift(ident, dy * step, dx * step, -1) == ident) & omask
                cosine = (nrm * on).sum(-1)
                distance = _plane(_shift(pos, dy * step, dx * step)[..., :3] - pos[..., :3], nrm, on)
                ok &= (cosine > 0.97) & (distance <= tolerance)
                weight = kernel[dx + 2] * kernel[dy + 2] * cosine.clamp_min(0) ** 32 * torch.exp(-distance / scale)
                s = (2.0 * (meta[..., 1].clamp_min(0) + om[..., 1]).clamp_min(0).sqrt()).clamp_min(0.02)
                edge = torch.exp(-(_luminance(v) - centre_l).abs() / s)
                weight = torch.where(meta[..., 0] > 0, weight * edge, weight) * ok
                total, weights = total + v[..., :3] * weight[..., None], weights + weight
        some = weights > 0.00001
        value = torch.where(some[..., None], total / weights.clamp_min(1e-30)[..., None], image[..., :3])
        outdepth = torch.where(light | (meta[..., 0] > 0) | some, depth, 0.0)
        image = torch.cat([value, outdepth[..., None]], -1)
        image[depth <= 0] = 0.0
        mask = (outdepth > 0) & (depth > 0)
    return image
