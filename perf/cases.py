"""The work that a program built on this library has it do, as timed cases.

A case is a dict of plain values; its "kind" says which of the library's
public entry points a pass goes through:

* frame      the drop-in call of the reference's host code: one view into a
             host image (octree_glc_update)
* batch      several views into device buffers in one call (qbc_render_views)
* character  the per-frame work of an animated scene: skin the character,
             rebuild its tree, take its normals, render (qbc_dynamic_update_run
             + qbc_render_views, or the same frame as a captured graph)
* twopass    the two-pass frame, plain or with the occluder network's
             proposals (qbc_render_views_ex)
* rays       batched ray queries (qbc_trace_rays)
* load       a level load: bulk build of the static tree from points, model
             upload, first frame (qbc_build_tree, qbc_upload_device)
* edit       a level restored from its node array, shot at and drawn again
             (qbc_upload_device, qbc_tree_remove_points)
* gradient   one gradient of the occluder network's training
* eval       the occluder network's outputs for a table of features

Scenes are seeded points on a floor or room with boxes and spheres, as the
library's own synthetic scenes are, made on the GPU in octree order.
"""
import ctypes as C
import math

import numpy as np
import torch

import qubatron_gb300 as qb
from qubatron_gb300 import _lib, scenes
from qubatron_gb300.octree_glc import view_setup

S = 1800.0
LEVELS = 12
CHARACTER_ROOT = (900.0, 500.0, 1100.0)
BONES = 12


def listed():
    return [
        # the host program's draw call at its smallest: latency and launches
        {"name": "frame_320x240", "kind": "frame", "scene": "floor", "points": 200_000, "w": 320, "h": 240},
        # the reference's default window over a mid-size level
        {"name": "frame_1200x800", "kind": "frame", "scene": "room", "points": 5_000_000, "w": 1200, "h": 800},
        # a camera path over a room-scale level, the benchmark's own batch
        {"name": "batch_room_16x1080p", "kind": "batch", "scene": "room", "points": 20_000_000, "views": 16,
         "w": 1920, "h": 1080, "streams": "rgba8"},
        # every per-pixel stream (colour, flags, leaf, intersection, visits) of odd-sized views
        {"name": "batch_streams_odd", "kind": "batch", "scene": "floor", "points": 1_000_000, "views": 3,
         "w": 1021, "h": 577, "streams": "all"},
        # a game frame: a large animated character, views of mixed sizes, replayed as a graph
        {"name": "character_2m_mixed", "kind": "character", "points": 1_000_000, "char": 2_000_000, "views": 12,
         "graph": True},
        # a small character and one view, queued call by call: rebuild latency
        {"name": "character_50k", "kind": "character", "points": 200_000, "char": 50_000, "views": 1, "graph": False},
        # shadow rays behind the occluder network
        {"name": "twopass_mlp_4x1080p", "kind": "twopass", "scene": "floor", "points": 1_000_000, "views": 4,
         "w": 1920, "h": 1080, "mlp": True},
        # the game logic's line-of-sight queries, host arrays
        {"name": "rays_host_1000", "kind": "rays", "scene": "room", "points": 1_000_000, "n": 1000, "host": True},
        # particle collisions: millions of incoherent rays in device memory
        {"name": "rays_device_4m", "kind": "rays", "scene": "room", "points": 5_000_000, "n": 4_000_000,
         "host": False},
        # a room-scale level load
        {"name": "load_20m", "kind": "load", "scene": "room", "points": 20_000_000, "w": 1280, "h": 720},
        # a level restored and edited by 20000 removals
        {"name": "edit_1m", "kind": "edit", "scene": "floor", "points": 1_000_000, "removals": 20_000, "w": 1280,
         "h": 720},
        # one minibatch of network training
        {"name": "gradient_8192", "kind": "gradient", "rows": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "batch", "batch", "character", "twopass", "rays", "load", "edit", "gradient", "eval"])
    scene = rng.choice(["floor", "room"])
    if kind == "frame":
        return {"kind": kind, "scene": scene, "points": _log(rng, 50_000, 5_000_000), "w": _log(rng, 160, 1920),
                "h": _log(rng, 120, 1080)}
    if kind == "batch":
        return {"kind": kind, "scene": scene, "points": _log(rng, 100_000, 20_000_000), "views": rng.randint(1, 16),
                "w": _log(rng, 160, 1920), "h": _log(rng, 120, 1080), "streams": rng.choice(["rgba8", "rgba8", "all"])}
    if kind == "character":
        return {"kind": kind, "points": _log(rng, 100_000, 1_000_000), "char": _log(rng, 20_000, 2_000_000),
                "views": rng.randint(1, 12), "graph": rng.choice([True, False])}
    if kind == "twopass":
        return {"kind": kind, "scene": scene, "points": _log(rng, 100_000, 5_000_000), "views": rng.randint(1, 4),
                "w": _log(rng, 160, 1920), "h": _log(rng, 120, 1080), "mlp": rng.choice([True, False])}
    if kind == "rays":
        host = rng.choice([True, False])
        return {"kind": kind, "scene": scene, "points": _log(rng, 100_000, 5_000_000),
                "n": _log(rng, 1, 16_384) if host else _log(rng, 1_000, 4_000_000), "host": host}
    if kind == "load":
        return {"kind": kind, "scene": scene, "points": _log(rng, 10_000, 20_000_000), "w": _log(rng, 160, 1280),
                "h": _log(rng, 120, 720)}
    if kind == "edit":
        return {"kind": kind, "scene": scene, "points": _log(rng, 50_000, 1_000_000),
                "removals": _log(rng, 1, 100_000), "w": _log(rng, 160, 1280), "h": _log(rng, 120, 720)}
    return {"kind": kind, "rows": _log(rng, 64, 65_536)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _primitives(kind, rng):
    """(rects [n, 12]: origin, u, v, normal; spheres [m, 4]; colours) of a scene."""
    rects = []
    if kind == "floor":
        lo, hi, floor, top = 0.0, S, 0.05 * S, S
        rects.append(((0.0, floor, 0.0), (S, 0, 0), (0, 0, S), (0, 1, 0)))
        boxes, spheres, bs, ss = 40, 20, (50.0, 400.0), (30.0, 200.0)
    else:
        m, w, h = 0.02 * S, 0.96 * S, 0.6 * S
        lo, hi, floor, top = m, S - m, m, m + h
        rects += [((m, m, m), (w, 0, 0), (0, 0, w), (0, 1, 0)), ((m, m + h, m), (w, 0, 0), (0, 0, w), (0, -1, 0)),
                  ((m, m, m), (0, h, 0), (0, 0, w), (1, 0, 0)), ((S - m, m, m), (0, h, 0), (0, 0, w), (-1, 0, 0)),
                  ((m, m, m), (w, 0, 0), (0, h, 0), (0, 0, 1)), ((m, m, S - m), (w, 0, 0), (0, h, 0), (0, 0, -1))]
        boxes, spheres, bs, ss = 200, 100, (20.0, 300.0), (10.0, 150.0)
    colour = [tuple(rng.uniform(0.0, 1.0, 3)) for _ in rects]
    for _ in range(boxes):
        sx, sy, sz = rng.uniform(bs[0], bs[1], 3)
        x, z = rng.uniform(lo, hi - sx), rng.uniform(lo, hi - sz)
        y = floor
        rects += [((x, y + sy, z), (sx, 0, 0), (0, 0, sz), (0, 1, 0)), ((x, y, z + sz), (sx, 0, 0), (0, sy, 0), (0, 0, 1)),
                  ((x, y, z), (sx, 0, 0), (0, sy, 0), (0, 0, -1)), ((x, y, z), (0, sy, 0), (0, 0, sz), (-1, 0, 0)),
                  ((x + sx, y, z), (0, sy, 0), (0, 0, sz), (1, 0, 0))]
        colour += [tuple(rng.uniform(0.0, 1.0, 3))] * 5
    balls = []
    for _ in range(spheres):
        r = rng.uniform(*ss)
        balls.append((rng.uniform(lo + r, hi - r), rng.uniform(floor + r, top - r), rng.uniform(lo + r, hi - r), r))
        colour.append(tuple(rng.uniform(0.0, 1.0, 3)))
    return rects, balls, colour


def _octree_order(p):
    """Order of points by their octree cell at the deepest level, root first."""
    cell = (p * (4096.0 / S)).to(torch.int64).clamp_(0, 4095)
    key = torch.zeros(p.shape[0], dtype=torch.int64, device=p.device)
    for level in range(LEVELS - 1, -1, -1):
        for axis in (2, 1, 0):
            bit = (cell[:, axis] >> level) & 1
            key = (key << 1) | (bit if axis == 0 else 1 - bit)
    return torch.argsort(key)


def _points(kind, n, seed):
    """n float32 points, normals and colours of a scene, on the GPU in octree order."""
    rects, balls, colour = _primitives(kind, np.random.RandomState(seed % (1 << 32)))
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(seed)
    r = torch.tensor([sum(map(list, q), []) for q in rects], dtype=torch.float32, device=dev)
    b = torch.tensor(balls, dtype=torch.float32, device=dev)
    col = torch.tensor(colour, dtype=torch.float32, device=dev)
    area = torch.cat([r[:, 3:6].norm(dim=1) * r[:, 6:9].norm(dim=1), 4.0 * math.pi * b[:, 3] ** 2])
    cdf = torch.cumsum(area.double(), 0)
    pick = torch.searchsorted(cdf, torch.rand(n, generator=g, device=dev, dtype=torch.float64) * cdf[-1])
    pick.clamp_(max=area.numel() - 1)
    nr = r.shape[0]
    q = r[pick.clamp(max=nr - 1)]
    uv = torch.rand(n, 2, generator=g, device=dev)
    p = q[:, 0:3] + uv[:, :1] * q[:, 3:6] + uv[:, 1:] * q[:, 6:9]
    nrm = q[:, 9:12].clone()
    on_ball = pick >= nr
    s = b[(pick - nr).clamp(min=0)]
    d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device=dev), dim=1)
    p = torch.where(on_ball[:, None], s[:, :3] + s[:, 3:] * d, p)
    nrm = torch.where(on_ball[:, None], d, nrm)
    c = col[pick] + (0.05 * (2.0 * torch.rand(n, 3, generator=g, device=dev) - 1.0) if kind == "room" else 0.0)
    p.clamp_(0.0, 1799.99)
    order = _octree_order(p)
    return p[order].contiguous(), nrm[order].contiguous(), c.clamp_(0.0, 1.0)[order].contiguous()


def _upload(ctx, t, buftype):
    ctx.upload_device(t.data_ptr(), qb.GL_FLOAT, t.numel() * 4, 12, 0, t.numel() * 4, buftype)


def _static(ctx, kind, n, seed):
    p, nrm, col = _points(kind, n, seed)
    torch.cuda.synchronize()
    _upload(ctx, col, qb.OCTREE_GLC_BUFFER_STATIC_COLOR)
    _upload(ctx, nrm, qb.OCTREE_GLC_BUFFER_STATIC_NORMAL)
    ctx.build_tree(False, (p.data_ptr(), n), S, LEVELS)
    ctx.synchronize()
    return p


def _character(n, seed):
    """Rest points, normals, colours, bone of each point and joints of a chain of capsules."""
    rng = np.random.RandomState(seed % (1 << 32))
    joints = [np.array(CHARACTER_ROOT)]
    for _ in range(BONES):
        d = np.array([rng.uniform(-0.4, 0.4), 1.0, rng.uniform(-0.4, 0.4)])
        joints.append(joints[-1] + 40.0 * d / np.linalg.norm(d))
    joints = np.array(joints)
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(seed + 1)
    j = torch.tensor(joints, dtype=torch.float32, device=dev)
    bone = torch.randint(0, BONES, (n,), generator=g, device=dev, dtype=torch.int32)
    a, e = j[bone.long()], j[bone.long() + 1]
    axis = torch.nn.functional.normalize(e - a, dim=1)
    d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device=dev), dim=1)
    radial = torch.nn.functional.normalize(d - (d * axis).sum(1, keepdim=True) * axis, dim=1)
    side = torch.rand(n, 1, generator=g, device=dev) < 40.0 / (40.0 + 2 * 12.0)
    t = torch.rand(n, 1, generator=g, device=dev)
    end = torch.where((d * axis).sum(1, keepdim=True) > 0, e, a)
    p = torch.where(side, a + t * (e - a) + 12.0 * radial, end + 12.0 * d).contiguous()
    nrm = torch.where(side, radial, d).contiguous()
    col = torch.rand(BONES, 3, generator=g, device=dev)[bone.long()].contiguous()
    return p, nrm, col, bone, scenes.Character(None, None, None, None, joints)


def _buffers(views, streams):
    """Device outputs: one flat tensor per stream over all views, and the
    per-view output pointers into them."""
    per = {"rgba8": (4, torch.uint8), "rgba32f": (4, torch.float32), "flags": (1, torch.int32),
           "leaf": (4, torch.int32), "isp": (4, torch.float32), "visits": (4, torch.int32)}
    px = [v.width_px * v.height_px for v in views]
    arrays, outs = {}, [_lib.Outputs() for _ in views]
    for s in streams:
        comps, dt = per[s]
        a = torch.zeros(sum(px) * comps, dtype=dt, device="cuda")
        at = a.data_ptr()
        for o, n in zip(outs, px):
            setattr(o, s, at)
            at += n * comps * a.element_size()
        arrays[s] = a
    return arrays, outs


def _views(seed, n, w, h):
    return [view_setup(w, h, pos, ang, 0.0, 10, LEVELS, S, 0, scenes.vertical_fov_focal(h))
            for pos, ang in scenes.spline_poses(seed, n)]


def _network(seed):
    """Parameters like a trained network's: uniform weights, outputs spread over (0, 1)."""
    rng = np.random.RandomState((seed + 77) % (1 << 32))
    p = []
    for fan, rows, used_in, used_out in ((48, 128, 45, 128), (128, 128, 128, 128), (128, 128, 128, 128),
                                         (128, 16, 128, 4)):
        w = rng.uniform(-1.7, 1.7, (rows, fan)) / math.sqrt(used_in)
        w[used_out:] = 0.0
        w[:, used_in:] = 0.0
        bias = np.zeros(rows)
        if rows == 16:
            bias[:4] = (0.2, 0.5, 0.8, 0.1)
        p += [w.ravel(), bias]
    return np.concatenate(p).astype(np.float32)


def _features(m, seed):
    """Feature rows of shaded pixels, and the labels of logged shadow walks."""
    rng = np.random.RandomState((seed + 5) % (1 << 32))
    hit = rng.uniform(0.0, 1.0, (m, 3))
    n, to_light = rng.normal(size=(m, 3)), rng.normal(size=(m, 3))
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    to_light /= np.linalg.norm(to_light, axis=1, keepdims=True)
    cols = [hit, n, to_light]
    for q in range(6):
        a = math.pi * (4 << q) * hit
        cols.append(np.stack([np.sin(a), np.cos(a)], 2).reshape(m, 6))
    kind = (rng.uniform(size=m) < 0.4).astype(np.int8)
    t = np.where(kind == 1, rng.uniform(0.0, 1.0, m), 2.0)
    return np.concatenate(cols, 1).astype(np.float32), t.astype(np.float32), kind


def prepare(case, seed):
    k = case["kind"]
    ctx = qb.octree_glc_init(device=0)
    s = {"case": case, "ctx": ctx}
    if k in ("gradient", "eval"):
        s["x"], s["t"], s["label"] = _features(case["rows"], seed)
        ctx.proposal_set_params(_network(seed))
    elif k == "frame":
        _static(ctx, case["scene"], case["points"], seed)
        s["pos"], s["ang"] = scenes.spline_poses(seed, 1)[0]
    elif k in ("batch", "twopass"):
        _static(ctx, case["scene"], case["points"], seed)
        s["views"] = _views(seed, case["views"], case["w"], case["h"])
        every = ("rgba8", "rgba32f", "flags", "leaf", "isp", "visits")
        s["out"], s["outs"] = _buffers(s["views"], every if case.get("streams") == "all" else ("rgba8",))
        if case.get("mlp"):
            ctx.proposal_set_params(_network(seed))
    elif k == "character":
        _static(ctx, "floor", case["points"], seed)
        p, nrm, col, bone, ch = _character(case["char"], seed)
        s["keep"] = (p, nrm, col, bone)
        s["bones"] = torch.tensor(scenes.pose_bones(ch, seed % 1000), device="cuda")
        s["pnts"], s["nrms"] = torch.empty_like(p), torch.empty_like(nrm)
        torch.cuda.synchronize()
        _upload(ctx, col, qb.OCTREE_GLC_BUFFER_DYNAMIC_COLOR)
        u = _lib.DynamicUpdate()
        u.rest_pnts, u.rest_nrms, u.bone, u.bones = p.data_ptr(), nrm.data_ptr(), bone.data_ptr(), s["bones"].data_ptr()
        u.pnts, u.nrms, u.n, u.n_bones, u.levels, u.basesize = (s["pnts"].data_ptr(), s["nrms"].data_ptr(), case["char"],
                                                                BONES, LEVELS, S)
        s["update"] = u
        # sizes of a split-screen and capture mix, one of each in turn
        mix = [(1920, 1080), (1280, 720), (640, 480), (320, 240)]
        _, poses = scenes.batch_views(seed, case["views"])
        s["views"] = [view_setup(w, h, pos, ang, 0.0, 10, LEVELS, S, 0, scenes.vertical_fov_focal(h))
                      for (w, h), (pos, ang) in zip((mix * case["views"])[: case["views"]], poses)]
        s["out"], s["outs"] = _buffers(s["views"], ("rgba8",))
        if case["graph"]:
            s["graph"] = ctx.graph_capture_dynamic(u, s["views"], s["outs"])
    elif k == "rays":
        _static(ctx, case["scene"], case["points"], seed)
        n = case["n"]
        g = torch.Generator(device="cuda").manual_seed(seed + 3)
        pos = (torch.rand(n, 3, generator=g, device="cuda") * (0.5 * S) + 0.1 * S).contiguous()
        d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device="cuda"), dim=1).contiguous()
        if case["host"]:
            s["pos"], s["dir"] = pos.cpu().numpy(), d.cpu().numpy()
        else:
            s["pos"], s["dir"] = pos, d
            s["out"] = {"status": torch.zeros(n, dtype=torch.int32, device="cuda"),
                        "leaf": torch.zeros(n, 2, dtype=torch.int32, device="cuda"),
                        "isp": torch.zeros(n, 4, device="cuda"), "nrm": torch.zeros(n, 4, device="cuda")}
    elif k == "load":
        s["p"], s["nrm"], s["col"] = _points(case["scene"], case["points"], seed)
        s["views"] = _views(seed, 1, case["w"], case["h"])
        s["out"], s["outs"] = _buffers(s["views"], ("rgba8", "leaf"))
    elif k == "edit":
        p = _static(ctx, case["scene"], case["points"], seed)
        s["nodes"] = torch.from_numpy(ctx.download_tree(False)).cuda()
        pick = np.random.RandomState(seed % (1 << 32)).randint(0, case["points"], case["removals"])
        s["shots"] = p.cpu().numpy()[pick]
        s["views"] = _views(seed, 1, case["w"], case["h"])
        s["out"], s["outs"] = _buffers(s["views"], ("rgba8", "leaf"))
    torch.cuda.synchronize()
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    k = case["kind"]
    if k == "frame":
        return qb.octree_glc_update(ctx, case["w"], case["h"], s["pos"], s["ang"], 0.0, 10, LEVELS, S)
    if k == "batch":
        ctx.render_views(s["views"], s["outs"], True)
        return s["out"]
    if k == "character":
        if case["graph"]:
            s["graph"].launch()
        else:
            ctx.dynamic_update(s["update"])
            ctx.render_views(s["views"], s["outs"], True)
        return {"rgba8": s["out"]["rgba8"], "pnts": s["pnts"], "nrms": s["nrms"]}
    if k == "twopass":
        ctx.render_views_ex(s["views"], s["outs"], True, two_pass=True,
                            proposals=_lib.PROPOSE_MLP if case["mlp"] else _lib.PROPOSE_NONE)
        return s["out"]
    if k == "rays":
        bc = (0.0, S, S, S)
        if case["host"]:
            return ctx.trace_rays(s["pos"], s["dir"], bc, LEVELS)
        o = s["out"]
        h = _lib.RayHits(status=o["status"].data_ptr(), leaf=o["leaf"].data_ptr(), isp=o["isp"].data_ptr(),
                         nrm=o["nrm"].data_ptr())
        _lib.check(_lib.load().qbc_trace_rays(ctx.handle, C.c_void_p(s["pos"].data_ptr()),
                                              C.c_void_p(s["dir"].data_ptr()), case["n"], (C.c_float * 4)(*bc), LEVELS,
                                              C.byref(h), 1))
        return o
    if k == "load":
        _upload(ctx, s["col"], qb.OCTREE_GLC_BUFFER_STATIC_COLOR)
        _upload(ctx, s["nrm"], qb.OCTREE_GLC_BUFFER_STATIC_NORMAL)
        nodes = ctx.build_tree(False, (s["p"].data_ptr(), case["points"]), S, LEVELS)
        ctx.render_views(s["views"], s["outs"], True)
        return {"nodes": nodes, **s["out"]}
    if k == "edit":
        n = s["nodes"]
        ctx.upload_device(n.data_ptr(), qb.GL_INT, n.numel() * 4, 16, 0, n.numel() * 4,
                          qb.OCTREE_GLC_BUFFER_STATIC_OCTREE)
        model, parent, removed = ctx.remove_points(False, s["shots"], S, LEVELS)
        ctx.render_views(s["views"], s["outs"], True)
        return {"model": model, "parent": parent, "removed": removed, **s["out"]}
    if k == "gradient":
        loss, grad = ctx.proposal_gradient(s["x"], s["t"], s["label"])
        return {"loss": loss, "grad": grad}
    return ctx.proposal_eval(s["x"])


def work(case):
    """Bytes of each input read and output written once, and the operations of
    the shortest walk: per ray one subnode test (about 60 operations) on each
    level down to its leaf, that leaf's block, model index, texel and normal."""
    k = case["kind"]
    ray_ops, ray_bytes = 60 * LEVELS, 64

    def frame(px, out):
        return {"bytes": px * (2 * ray_bytes + out), "flops": 2 * px * ray_ops}

    if k == "frame":
        return frame(case["w"] * case["h"], 4)
    if k in ("batch", "twopass"):
        px = case["views"] * case["w"] * case["h"]
        w = frame(px, 72 if case.get("streams") == "all" else 4)
        if case.get("mlp"):
            w["flops"] += 2 * px * 40960
        return w
    if k == "character":
        mix = [1920 * 1080, 1280 * 720, 640 * 480, 320 * 240]
        w = frame(sum((mix * case["views"])[: case["views"]]), 4)
        n = case["char"]
        # skin (points, normals and bones in, points and normals out), about 2.6 nodes a point out
        w["bytes"] += n * (52 + 16) + 2.6 * n * 100
        w["flops"] += n * (33 + 12 * LEVELS)
        return w
    if k == "rays":
        return {"bytes": case["n"] * (24 + 44 + ray_bytes), "flops": case["n"] * ray_ops}
    if k in ("load", "edit"):
        w = frame(case["w"] * case["h"], 20)
        n = case["points"]
        # points and attributes in, attributes and about 2.6 nodes a point out; an edit reads the node array
        w["bytes"] += n * (36 + 32) + 2.6 * n * 100 if k == "load" else 2.6 * n * (48 + 100) + case["removals"] * 20
        w["flops"] += n * 12 * LEVELS
        return w
    macs = 45 * 128 + 2 * 128 * 128 + 128 * 4
    m = case["rows"]
    if k == "gradient":
        return {"bytes": m * (180 + 5) + 2 * 4 * 41360, "flops": 6 * m * macs}
    return {"bytes": m * (180 + 16) + 4 * 41360, "flops": 2 * m * macs}


def exact(case, seed):
    k = case["kind"]
    if k == "character":
        p, nrm, _, bone, ch = _character(case["char"], seed)
        m = torch.tensor(scenes.pose_bones(ch, seed % 1000), device="cuda").double()[bone.long()]
        rot, t = m[:, :9].reshape(-1, 3, 3), m[:, 9:]
        return {"rgba8": None, "pnts": (rot @ p.double()[:, :, None])[:, :, 0] + t,
                "nrms": (rot @ nrm.double()[:, :, None])[:, :, 0]}
    if k not in ("gradient", "eval"):
        return None
    x, t, label = (torch.from_numpy(a).cuda() for a in _features(case["rows"], seed))
    flat = torch.from_numpy(_network(seed)).cuda().double()
    parts, at = [], 0
    for shape in ((128, 48), (128,), (128, 128), (128,), (128, 128), (128,), (16, 128), (16,)):
        n = math.prod(shape)
        parts.append(flat[at:at + n].reshape(shape).clone().requires_grad_(True))
        at += n
    a = torch.nn.functional.pad(x.double(), (0, 3))
    for layer in range(3):
        a = torch.nn.functional.gelu(a @ parts[2 * layer].T + parts[2 * layer + 1])
    o = a @ parts[6].T + parts[7]
    if k == "eval":
        return o[:, :4].detach()
    # the training loss: winner-take-all distance of the three outputs for
    # occluded rows, a hinge past 1.1 for lit ones, cross-entropy on the gate
    occluded = (label == 1).double()
    d = o[:, :3] - t.double()[:, None]
    weight = torch.full_like(d, 0.02).scatter_(1, d.abs().argmin(1, keepdim=True), 1.0)
    loss = occluded * (weight * d * d).sum(1) + (1 - occluded) * (0.5 * (1.1 - o[:, :3]).clamp(min=0) ** 2).sum(1)
    loss = loss + 0.05 * torch.nn.functional.binary_cross_entropy_with_logits(o[:, 3], occluded, reduction="none")
    loss = loss.mean()
    loss.backward()
    return {"loss": float(loss), "grad": torch.cat([q.grad.reshape(-1) for q in parts])}
