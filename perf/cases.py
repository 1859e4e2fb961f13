"""What the renderer is measured on: the calls that its programs make, through
the package's public entry points, over the range of scenes, films and surfel
counts that its own scene files, tests and benchmark use.

A case is a dict of plain values; `kind` says which call it is:

  frame     Context.frame: one whole frame of a scene whose surfels are in
            place (transfer build, light, solve, grid, shading, encode).
  view      Context.render_frame: another camera on a solved scene, as a
            viewer or a turntable renders it.
  generate  Context.generate and the surfels read back: the start of any
            program with a new scene.
  solve     solve_noalloc on device buffers of the caller: the Jacobi solve
            inside an engine that owns its memory.
  relight   Context.solve_batched: many light settings solved on one transfer.
  gradient  Context.diff_forward and diff_backward: a step of an optimiser
            over surfel albedo and light emission.
  path      Context.render_reference: the path-traced check image.
  packed    MultiScene.run and the frames read back: many scenes in one launch.
"""
import math

import numpy as np
import torch

import interflect_b200 as ifx
from interflect_b200.scenes import gen_scenes


# ------------------------------------------------------------------- cases ----
def listed():
    return [
        # The smallest call: a thumbnail of a few objects, all launches and latency.
        {"name": "frame_thumbnail", "kind": "frame", "scene": "stress", "prims": 9, "surfels": 1500, "width": 97,
         "height": 61, "cluster_res": 4, "mode": "beauty"},
        # The benchmark's Cornell box at its own size, the common test image.
        {"name": "frame_cornell", "kind": "frame", "scene": "cornell", "prims": 0, "surfels": 20000, "width": 260,
         "height": 260, "cluster_res": 8, "mode": "beauty"},
        # The product shot at full HD, the benchmark's default workload.
        {"name": "frame_product", "kind": "frame", "scene": "product", "prims": 0, "surfels": 200000, "width": 1920,
         "height": 1080, "cluster_res": 8, "mode": "beauty"},
        # Hundreds of objects (the stress recipe) at an odd film size: a large BVH, tens of millions of cones.
        {"name": "frame_stress", "kind": "frame", "scene": "stress", "prims": 512, "surfels": 50000, "width": 961,
         "height": 541, "cluster_res": 8, "mode": "beauty"},
        # A turntable step: only the camera moves, the solved scene is kept; the film comes back linear too.
        {"name": "view_turntable", "kind": "view", "scene": "product_strict", "prims": 0, "surfels": 20000,
         "width": 853, "height": 479, "cluster_res": 8, "mode": "beauty"},
        # A new scene's surfels at the product shot's density.
        {"name": "generate_product", "kind": "generate", "scene": "product", "prims": 0, "surfels": 200000},
        # The solve in an engine's own buffers: a small room between two frames, and the stress scene's size.
        {"name": "solve_room", "kind": "solve", "n": 12270, "cells": 7, "keep": 0.04, "bounces": 16},
        {"name": "solve_million", "kind": "solve", "n": 1000000, "cells": 16, "keep": 0.085, "bounces": 24},
        # Light settings of an animation or a lookup table, sources from the host and results back to it.
        {"name": "relight_batch", "kind": "relight", "n": 20000, "res": 8, "keep": 0.35, "rhs": 64, "bounces": 12},
        # One optimiser step on the benchmark's differentiation scene.
        {"name": "gradient_step", "kind": "gradient", "scene": "cornell_fill", "prims": 0, "surfels": 20000,
         "width": 512, "height": 512, "cluster_res": 8, "bounces": 12},
        # The path-traced check image at a preview's sample count.
        {"name": "path_reference", "kind": "path", "scene": "cornell_strict", "prims": 0, "width": 150, "height": 150,
         "spp": 48},
        # Scenes of mixed sizes solved and composed in one launch (a data set's or a service's batch).
        {"name": "packed_scenes", "kind": "packed", "scenes": 6, "prims": 40, "surfels": 12000, "side": 448,
         "bounces": 24},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "view", "generate", "solve", "solve", "relight", "gradient", "path",
                       "packed"])
    if kind in ("frame", "view"):
        scene = rng.choice(["stress", "cornell", "product", "product_strict"])
        prims = _log(rng, 8, 512) if scene == "stress" else 0
        return {"kind": kind, "scene": scene, "prims": prims, "surfels": _log(rng, 1500, 40000),
                "width": _log(rng, 90, 1000), "height": _log(rng, 60, 600), "cluster_res": rng.choice([4, 6, 8]),
                "mode": rng.choice(["beauty", "beauty", "beauty", "indirect", "direct"])}
    if kind == "generate":
        scene = rng.choice(["stress", "cornell", "product"])
        return {"kind": kind, "scene": scene, "prims": _log(rng, 8, 128) if scene == "stress" else 0,
                "surfels": _log(rng, 2000, 200000)}
    if kind == "solve":
        return {"kind": kind, "n": _log(rng, 2000, 800000), "cells": rng.randint(4, 14),
                "keep": round(rng.uniform(0.03, 0.12), 3), "bounces": rng.choice([8, 12, 16, 24])}
    if kind == "relight":
        return {"kind": kind, "n": _log(rng, 2000, 20000), "res": rng.choice([4, 6, 8]),
                "keep": round(rng.uniform(0.1, 0.4), 3), "rhs": _log(rng, 3, 64), "bounces": rng.choice([8, 12, 16])}
    if kind == "gradient":
        side = _log(rng, 64, 512)
        return {"kind": kind, "scene": "cornell_fill", "prims": 0, "surfels": _log(rng, 3000, 20000), "width": side,
                "height": max(1, side - rng.randint(0, 9)), "cluster_res": rng.choice([4, 8]),
                "bounces": rng.randint(4, 14)}
    if kind == "path":
        return {"kind": kind, "scene": rng.choice(["cornell_strict", "cornell", "product_strict"]), "prims": 0,
                "width": _log(rng, 40, 160), "height": _log(rng, 40, 160), "spp": _log(rng, 8, 48)}
    return {"kind": kind, "scenes": rng.randint(2, 6), "prims": _log(rng, 8, 60), "surfels": _log(rng, 2000, 12000),
            "side": 64 * rng.randint(3, 7), "bounces": rng.choice([12, 16, 24])}


# ------------------------------------------------------------------ scenes ----
def _scene_text(case, rng):
    """The case's scene with its movable parts placed by the seed. Surfel
    generation keeps the parts where they are and takes other colours, so that
    the number of surfels is the case's."""
    name = case["scene"]
    if case["kind"] == "generate":
        still = dict(case, kind="frame")
        return "\n".join(
            "%salbedo: [%.4g, %.4g, %.4g]%s" % (line.split("albedo: [")[0], *rng.uniform(0.2, 0.9, 3),
                                               line.split("albedo: [")[1].split("]", 1)[1])
            if "albedo: [" in line else line
            for line in _scene_text(still, np.random.default_rng(20261203)).splitlines()) + "\n"
    if name == "stress":
        return gen_scenes.stress_scene(rng, "stress", "random primitives", case["prims"], case.get("surfels", 1500),
                                       case.get("width", 320), case.get("height", 180), 24)
    text = {"cornell": lambda: gen_scenes.c1(True), "cornell_strict": lambda: gen_scenes.c1(False),
            "cornell_fill": gen_scenes.c5, "product": lambda: gen_scenes.c2(False),
            "product_strict": lambda: gen_scenes.c2(True)}[name]()
    lines = []
    for line in text.splitlines():
        # Spheres and tori without cut-outs stand a little elsewhere in each seed's scene.
        if line.startswith(("sphere {", "torus {")) and "subtract" not in line:
            head, rest = line.split("center: [", 1)
            xyz, tail = rest.split("]", 1)
            x, y, z = (float(v) for v in xyz.split(","))
            dx, dz = rng.uniform(-0.03, 0.03, 2)
            line = "%scenter: [%.6g, %.6g, %.6g]%s" % (head, x + dx, y, z + dz, tail)
        lines.append(line)
    return "\n".join(lines) + "\n"


def _camera(scene, angle):
    """The scene's camera turned about its target by `angle` (radians)."""
    cam = scene.info.camera
    p, q = np.array(cam["pos"], np.float64), np.array(cam["look"], np.float64)
    d, c, s = p - q, math.cos(angle), math.sin(angle)
    return ifx.camera((q[0] + c * d[0] + s * d[2], p[1], q[2] - s * d[0] + c * d[2]), cam["look"], cam["up"], cam["fov"])


def _placed(case, seed, transfer):
    """A context with the seed's scene and surfels in place, and (transfer) its solved light."""
    rng = np.random.default_rng(seed)
    scene = ifx.parse(_scene_text(case, rng))
    if "width" in case and "surfels" in case:
        scene.set_cfg(width=case["width"], height=case["height"], surfels=case["surfels"])
    ctx = ifx.Context()
    ctx.upload(scene)
    if "surfels" in case and case["kind"] != "generate":
        ctx.generate(case["surfels"])
        ctx.set_light_emission(ctx.light_emission() * rng.uniform(0.6, 1.4, (ctx.n_lights, 1)).astype(np.float32))
    if transfer:
        ctx.build(case["cluster_res"])
    return ctx, scene, rng


# -------------------------------------------------- the synthetic solve's room ----
def _room(n, cells, keep, seed, side=1.0):
    """A closed room's transfer as the solve sees one: n surfels on the six
    walls of [-side, side]^3 in random order, a cluster per cell of a cells x
    cells raster of each wall, and per surfel links to the clusters it sees (a
    share `keep` of them: the others are hidden, by source and target cluster
    alike) weighted by the disc form factor and calibrated to a row sum of at
    most 0.8. All made on the GPU in torch."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def rand(*shape):
        return torch.rand(*shape, generator=g, device="cuda")

    face = torch.randint(0, 6, (n,), generator=g, device="cuda")
    cell = torch.randint(0, cells * cells, (n,), generator=g, device="cuda")
    ncl = 6 * cells * cells
    # Every cluster has a member.
    face[:ncl], cell[:ncl] = torch.arange(ncl, device="cuda") // (cells * cells), torch.arange(ncl, device="cuda") % (cells * cells)
    order = torch.randperm(n, generator=g, device="cuda")
    face, cell = face[order], cell[order]
    # Positions stay clear of the cells' edges.
    u = ((cell // cells) + 0.1 + 0.8 * rand(n)) / cells * 2 - 1
    v = ((cell % cells) + 0.1 + 0.8 * rand(n)) / cells * 2 - 1
    axis, sign = face // 2, (face % 2).float() * 2 - 1
    p, nrm = torch.empty(n, 3, device="cuda"), torch.zeros(n, 3, device="cuda")
    for a in range(3):
        m = axis == a
        p[m, a], p[m, (a + 1) % 3], p[m, (a + 2) % 3] = sign[m] * side, u[m] * side, v[m] * side
        nrm[m, a] = -sign[m]
    area = (24.0 * side * side / n) * (0.8 + 0.4 * rand(n))
    albedo = 0.2 + 0.7 * rand(6, 3)[face]
    emit = albedo * (rand(ncl)[face * cells * cells + cell] ** 4 * 3.0 * (0.7 + 0.6 * rand(n)))[:, None]
    cid = face * cells * cells + cell
    # Sums in 64 bits: the order that atomics add in does not show.
    f64 = torch.float64
    carea = torch.zeros(ncl, dtype=f64, device="cuda").index_add_(0, cid, area.to(f64))
    cpos = torch.zeros(ncl, 3, dtype=f64, device="cuda").index_add_(0, cid, (p * area[:, None]).to(f64)) / carea[:, None]
    carea, cpos = carea.float(), cpos.float()
    cn = torch.zeros(ncl, 3, device="cuda").index_copy_(0, cid, nrm)
    seen = rand(ncl, ncl) < keep * 0.95
    counts, idx, w = [], [], []
    for i in range(0, n, 32768):
        d = cpos[None] - p[i:i + 32768, None]
        r2 = (d * d).sum(-1)
        d = d / r2.sqrt()[..., None]
        ci, cc = (d * nrm[i:i + 32768, None]).sum(-1), -(d * cn[None]).sum(-1)
        ff = ci * cc * carea / (math.pi * r2 + carea)
        link = (ci > 1e-3) & (cc > 1e-3) & (ff >= 2e-5) & (seen[cid[i:i + 32768]] | (rand(*ff.shape) < keep * 0.05))
        ff = torch.where(link, ff * (0.3 + 0.7 * rand(*ff.shape)), 0.0)
        total = ff.sum(1, keepdim=True)
        ff = ff * torch.where(total > 0, torch.clamp(0.8 / total, max=8.0), 1.0)
        counts.append(link.sum(1))
        idx.append(link.nonzero()[:, 1].to(torch.int32))
        w.append(ff[link])
    starts = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    starts[1:] = torch.cumsum(torch.cat(counts), 0)
    return {"p": p, "n": nrm, "area": area, "albedo": albedo, "emit": emit, "cid": cid, "carea": carea, "cpos": cpos,
            "starts": starts.to(torch.int32), "idx": torch.cat(idx), "w": torch.cat(w), "ncl": ncl}


def _four(x, w=None):
    out = torch.zeros(x.shape[0], 4, device="cuda")
    out[:, :3] = x
    if w is not None:
        out[:, 3] = w
    return out


def _solve64(room, emit, bounces):
    """The bounces in 64 bits: (irradiance, radiosity) once the change is below 1e-4 or after `bounces`."""
    n, f64 = room["cid"].numel(), torch.float64
    area, albedo, e = room["area"].to(f64), room["albedo"].to(f64), emit.to(f64)
    csum = torch.zeros(room["ncl"], dtype=f64, device="cuda").index_add_(0, room["cid"], area)
    m = torch.sparse_csr_tensor(room["starts"].long(), room["idx"].long(), room["w"].to(f64), (n, room["ncl"]))
    rad, irr = e.clone(), torch.zeros_like(e)
    for _ in range(bounces):
        mean = torch.zeros(room["ncl"], 3, dtype=f64, device="cuda").index_add_(0, room["cid"], rad * area[:, None])
        irr = m @ (mean / csum[:, None])
        new = e + albedo * irr
        change = (new - rad).abs().max()
        rad = new
        if change < 1e-4:
            break
    return irr, rad


# The relighting room: a box whose inner walls stand at +-1, so that its
# surfels fall into the clusters that the context forms by position.
_ROOM_RAD = (
    "render { width: 64, height: 64, surfels: 1000, bounces: 12, exposure: 1.0 }\n"
    "camera { pos: [0, 0, 0.9], look: [0, 0, 0], up: [0, 1, 0], fov: 60 }\n"
    'material "m" { albedo: [0.7, 0.7, 0.7], roughness: 0.9 }\n'
    + "".join('box { center: [%g, %g, %g], size: [%g, %g, %g], mat: "m" }\n' % (
        *[1.05 * s if a == k else 0 for k in range(3)], *[0.1 if a == k else 2.2 for k in range(3)])
        for a in range(3) for s in (-1, 1))
    + "light { verts: [[-0.2, 0.9, -0.2], [0.2, 0.9, -0.2], [0.2, 0.9, 0.2], [-0.2, 0.9, 0.2]], emit: [5, 5, 5] }\n")


def _relight_inputs(case, seed):
    room = _room(case["n"], case["res"], case["keep"], seed)
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 99)
    gains = torch.rand(case["rhs"], 6, 3, generator=g, device="cuda") * 1.5 + 0.05
    # Each light setting: the walls' sources dimmed and tinted by wall.
    face = room["cid"] // (room["ncl"] // 6)
    return room, room["emit"][None] * gains[:, face]


def _relight_context(case, room):
    """A context with the room's surfels, its clusters in the room's order and
    the room's transfer. The context numbers clusters by position and normal:
    read back from its cluster centres, the room's are renumbered to match."""
    scene = ifx.parse(_ROOM_RAD)
    ctx = ifx.Context()
    ctx.upload(scene)
    host = {k: room[k].cpu().numpy() for k in ("p", "n", "albedo", "area", "starts", "idx", "w", "cid")}
    # The context's raster covers the scene's bounds, so a wall's cells are not
    # its cells: the walls' positions are scaled within the cluster test only.
    lo, hi = (np.array(b, np.float64) for b in (scene.info.bounds_lo, scene.info.bounds_hi))
    ctx.upload_surfels(lo + (host["p"] * 0.999 + 1) / 2 * (hi - lo), host["n"], host["albedo"], host["area"])
    nc = ctx.build_clusters(case["res"])
    c = ctx.clusters(nc)
    if nc != room["ncl"]:
        raise RuntimeError("the room's clusters are not the context's")
    number = np.empty(nc, np.uint32)
    first = c["members"][c["offsets"][:-1]]
    number[host["cid"][first]] = np.arange(nc, dtype=np.uint32)
    idx = number[host["idx"]]
    # Links ascend within a row, as the transfer build leaves them.
    rows = np.repeat(np.arange(case["n"]), np.diff(host["starts"]))
    order = np.lexsort((idx, rows))
    ctx.upload_transfer(host["starts"], idx[order], host["w"][order])
    return ctx


# -------------------------------------------------------------- the calls ----
def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        ctx, scene, rng = _placed(case, seed, False)
        cam, film = _camera(scene, rng.uniform(-0.25, 0.25)), None
        if case["width"] * case["height"] >= 1 << 20:
            # A program that renders large frames keeps its page-locked film, as the benchmark does.
            film = torch.zeros((case["height"], case["width"], 3), dtype=torch.uint8, pin_memory=True).numpy()
        return {"case": case, "ctx": ctx, "cam": cam, "film": film}
    if kind == "view":
        ctx, scene, rng = _placed(case, seed, True)
        ctx.light_surfels()
        ctx.solve(scene.cfg.bounces)
        ctx.grid_build()
        return {"case": case, "ctx": ctx, "cam": _camera(scene, rng.uniform(-math.pi / 3, math.pi / 3))}
    if kind == "generate":
        return {"case": case, "ctx": _placed(case, seed, False)[0]}
    if kind == "solve":
        room = _room(case["n"], case["cells"], case["keep"], seed)
        count = torch.bincount(room["cid"], minlength=room["ncl"])
        ends = torch.cumsum(count, 0)
        return {"case": case, "p": _four(room["p"], room["area"]), "direct": _four(room["emit"]),
                "albedo": _four(room["albedo"]), "irr": torch.zeros(case["n"], 4, device="cuda"),
                "rad": torch.zeros(case["n"], 4, device="cuda"), "cp": _four(room["cpos"], room["carea"]),
                "ranges": torch.stack([ends - count, ends], 1).to(torch.int32).contiguous(),
                "members": torch.sort(room["cid"], stable=True)[1].to(torch.int32), "starts": room["starts"],
                "idx": room["idx"], "w": room["w"]}
    if kind == "relight":
        room, emit = _relight_inputs(case, seed)
        return {"case": case, "ctx": _relight_context(case, room), "E": emit.cpu().numpy()}
    if kind == "gradient":
        ctx, scene, rng = _placed(case, seed, True)
        ctx.diff_setup(case["width"], case["height"], case["bounces"], cam=_camera(scene, rng.uniform(-0.2, 0.2)))
        rho = np.clip(ctx.surfels()["albedo"] * rng.uniform(0.8, 1.1, (ctx.n_surfels, 1)), 0.02, 0.95)
        return {"case": case, "ctx": ctx, "rho": rho.astype(np.float32), "emit": ctx.light_emission(),
                "grad": rng.normal(0, 1e-5, (case["height"], case["width"], 3)).astype(np.float32)}
    if kind == "path":
        ctx, scene, rng = _placed(case, seed, False)
        ctx.render_reference(8, 8, 1)  # the sampler's table, made once per context
        return {"case": case, "ctx": ctx, "cam": _camera(scene, rng.uniform(-0.2, 0.2))}
    if kind == "packed":
        rng = np.random.default_rng(seed)
        ms, members = ifx.MultiScene(), []
        for side, surfels, prims in _packed_sizes(case):
            scene = ifx.parse(gen_scenes.stress_scene(rng, "packed", "packed", prims, surfels, side, side,
                                                      case["bounces"]))
            ctx = ifx.Context()
            ctx.upload(scene)
            ctx.generate(surfels)
            ctx.build(8)
            ms.add(ctx, side, side, case["bounces"])
            members.append(ctx)
        ms.build()
        return {"case": case, "ms": ms, "members": members}
    raise ValueError(kind)


def _packed_sizes(case):
    """(film side, surfels requested, objects) of each packed scene: from half to one and a half times the case's."""
    out = []
    for i in range(case["scenes"]):
        share = 0.5 + i / (case["scenes"] - 1)
        out.append((max(64, int(case["side"] * share) // 64 * 64), max(1000, int(case["surfels"] * share)),
                    max(8, int(case["prims"] * share))))
    return out


def run(state):
    case, ctx = state["case"], state.get("ctx")
    kind = case["kind"]
    if kind == "frame":
        f = ctx.frame(case["width"], case["height"], mode=case["mode"], cluster_res=case["cluster_res"],
                      cam=state["cam"], linear=state["film"] is None, out_srgb=state["film"])
        t = f["transfer"]
        return {"srgb": f["srgb"], "linear": f["linear"], "links": t.links, "candidates": t.candidates,
                "evals": t.evals + f["light_evals"] + f["shade_evals"], "bounces": f["solve"].iterations,
                "residual": f["solve"].residual, "row_sum": t.mean_row_sum}
    if kind == "view":
        linear, srgb, evals = ctx.render_frame(case["width"], case["height"], mode=case["mode"], cam=state["cam"])
        return {"linear": linear, "srgb": srgb, "evals": evals}
    if kind == "generate":
        ctx.generate(case["surfels"])
        s = ctx.surfels()
        return {k: s[k] for k in ("p", "n", "albedo", "area")}
    if kind == "solve":
        state["rad"].copy_(state["direct"])  # the solve starts from the emitted light
        stats = ifx.solve_noalloc(
            state["rad"].device.index, torch.cuda.current_stream().cuda_stream, case["n"], state["cp"].shape[0],
            *(state[k].data_ptr() for k in ("p", "direct", "albedo", "irr", "rad", "cp", "ranges", "members",
                                            "starts", "idx", "w")), case["bounces"])
        return {"irr": state["irr"], "rad": state["rad"], "bounces": stats.iterations, "residual": stats.residual}
    if kind == "relight":
        rad, irr, bounces, residual = ctx.solve_batched(state["E"], case["bounces"])
        return {"rad": rad, "irr": irr, "bounces": bounces, "residual": residual}
    if kind == "gradient":
        image = ctx.diff_forward(state["rho"], state["emit"])
        g_rho, g_emit = ctx.diff_backward(state["grad"])
        return {"image": image, "g_rho": g_rho, "g_emit": g_emit}
    if kind == "path":
        linear, srgb = ctx.render_reference(case["width"], case["height"], spp=case["spp"], cam=state["cam"])
        return {"linear": linear, "srgb": srgb}
    state["ms"].run()
    out = []
    for i in range(len(state["members"])):
        linear, srgb, stats = state["ms"].download(i)
        out.append((linear, srgb, stats.iterations, stats.residual))
    return out


# Distance queries per film pixel and per surfel requested (transfer and light),
# as the library's work counters give them at the listed sizes; a query cannot
# do without the nearest object's distance and the march's own step, some 45 FLOP.
_QUERIES = {"stress": (130, 17000), "cornell": (34, 4100), "cornell_strict": (34, 4100), "cornell_fill": (34, 4100),
            "product": (101, 350), "product_strict": (99, 350)}
_QUERY_FLOP = 45


def work(case):
    kind = case["kind"]
    if kind in ("frame", "view"):
        px = case["width"] * case["height"]
        per_px, per_surfel = _QUERIES[case["scene"]]
        gi = kind == "frame" and case["mode"] != "direct"
        queries = px * per_px + (case["surfels"] * per_surfel * (case["cluster_res"] / 8) ** 2 if gi else 0)
        return {"bytes": 48 * case["surfels"] + 15 * px, "flops": queries * _QUERY_FLOP}
    if kind == "generate":
        # Each of the 24 seeds per surfel asked for (at most 6M) is walked onto the surface: some 5 steps of 5 queries.
        return {"bytes": 40 * case["surfels"], "flops": min(24 * case["surfels"], 6000000) * 25 * _QUERY_FLOP}
    if kind == "solve":
        links = case["n"] * 5 * case["cells"] ** 2 * case["keep"]
        return {"bytes": 8 * links + (5 * 16 + 8) * case["n"], "flops": 6 * links * min(case["bounces"], 12)}
    if kind == "relight":
        links = case["n"] * 5 * case["res"] ** 2 * case["keep"]
        return {"bytes": 8 * links + 36 * case["n"] * case["rhs"],
                "flops": 6 * links * case["rhs"] * min(case["bounces"], 10)}
    if kind == "gradient":
        # Per pixel some 8 gather entries (16 B) and two lights' coefficients (16 B); per surfel some 118 links.
        px, n = case["width"] * case["height"], case["surfels"]
        return {"bytes": px * (24 + 8 * 16 + 32) + n * (118 * 16 + 64 * case["bounces"]),
                "flops": px * 8 * 12 + n * 118 * 12 * case["bounces"]}
    if kind == "path":
        # Some 140 queries a path (camera ray, bounces, their normals and shadow rays).
        px = case["width"] * case["height"]
        return {"bytes": 15 * px, "flops": px * case["spp"] * 140 * _QUERY_FLOP}
    px = sum(s * s for s, _, _ in _packed_sizes(case))
    n = sum(k for _, k, _ in _packed_sizes(case))
    # Per pixel the stored hit, form factors and visibilities and the two films; per surfel some 100 links.
    return {"bytes": px * (32 + 8 * 4 + 15) + n * (8 * 100 + 112), "flops": px * 600 + n * 100 * 6 * 14}


def exact(case, seed):
    """The solve and the relighting in 64 bits. The other calls march rays
    whose every stopping decision is a 32-bit comparison (a hit, a step count,
    a link, an accepted surfel), so a 64-bit march is another image; and
    restating the whole renderer's hundreds of millions of distance queries in
    plain torch takes minutes a case."""
    if case["kind"] == "solve":
        room = _room(case["n"], case["cells"], case["keep"], seed)
        irr, rad = _solve64(room, room["emit"], case["bounces"])
        zero = torch.zeros(case["n"], 1, dtype=torch.float64, device="cuda")
        return {"irr": torch.cat([irr, zero], 1), "rad": torch.cat([rad, zero], 1), "bounces": None, "residual": None}
    if case["kind"] == "relight":
        room, emit = _relight_inputs(case, seed)
        got = [_solve64(room, e, case["bounces"]) for e in emit]
        return {"rad": torch.stack([r for _, r in got]).cpu().numpy(),
                "irr": torch.stack([i for i, _ in got]).cpu().numpy(), "bounces": None, "residual": None}
    return None
