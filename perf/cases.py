"""The work that programs built on this package have it do, as measurable cases.

A case is a dict of plain values; its "kind" names the call it stands for:

  build   one tree build (LBVH or the higher-quality PLOC build) into a kept builder
  trace   one launch of rays, closest or any hit, over one of the tree forms
  ao      one ambient-occlusion frame; with "rebuild" the frame of a moving scene, which
          builds the tree, regroups it and renders
  pt      one progressive path-tracing pass and the packed image
  diff    one differentiable render and its path-replay adjoint
  batch   many meshes built in one launch chain and their rays drained by one kernel

listed() holds the measured cases, draw() gives further ones of the same ranges.
Scenes and rays are those of minimumlbvh_b200.scenes, seeded.
"""
import math

import numpy as np
import torch

import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

SEED_CAP = 1 << 31
MAX_TRIS = 4_194_304
MAX_RAYS = 1_048_576


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # a debug mesh or a moving prop: the smallest build, launches and latency
        dict(name="build_prop_1000", kind="build", builder="lbvh", scene="soup", n=1000, normal=False),
        # an ordinary scene rebuilt every frame
        dict(name="build_field_213k", kind="build", builder="lbvh", scene="field", quads=256, spheres=64, normal=False),
        # the largest scene: 4M triangles
        dict(name="build_soup_4m", kind="build", builder="lbvh", scene="soup", n=MAX_TRIS, normal=False),
        # the higher-quality build of a scene that is loaded once
        dict(name="ploc_field_213k", kind="build", builder="ploc", scene="field", quads=256, spheres=64, normal=False),
        # picking and probe rays: few rays, a small scene, the default walk
        dict(name="trace_probe_4099", kind="trace", form="plain", query="closest", rays="random", nrays=4099,
             scene="soup", n=20_011),
        # shadow rays over the 4-wide tree
        dict(name="shadow_wide_1m", kind="trace", form="wide", query="any", rays="random", nrays=1_000_003,
             scene="field", quads=256, spheres=64),
        # every other pixel's camera ray of a 1920x1080 frame over the quantised 4-wide tree
        dict(name="camera_qwide_4m", kind="trace", form="qwide", query="closest", rays="camera", w=1920, h=1080,
             scene="soup", n=MAX_TRIS),
        # an AO frame through the default call: 512x512, 16 rays of radius 0.25 per hit
        dict(name="ao_field_512", kind="ao", form="plain", rebuild=False, w=512, h=512, samples=16, radius=0.25,
             sobol=True, scene="field", quads=256, spheres=64),
        # a frame of a moving 4M-triangle scene: build, 4-wide regrouping, 1920x1080 with 64 AO rays per hit
        dict(name="ao_frame_4m", kind="ao", form="wide", rebuild=True, w=1920, h=1080, samples=64, radius=0.1,
             sobol=True, scene="soup", n=MAX_TRIS),
        # a progressive path-tracing pass through the default call
        dict(name="pt_field_512", kind="pt", walk="plain", w=512, h=512, sobol=True, scene="field", quads=256,
             spheres=64),
        # an optimisation step on per-triangle albedo: render and adjoint, 64 samples, 3 bounces
        dict(name="diff_field_512", kind="diff", w=512, h=512, spp=64, bounces=3, quads=256, spheres=64),
        # many uneven meshes: one build and one trace of all of them
        dict(name="batch_256", kind="batch", meshes=256, tri_lo=64, tri_hi=65_536, ray_lo=1024, ray_hi=262_144,
             counts_seed=7, query="closest"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_scene(rng, n_hi=MAX_TRIS):
    if rng.random() < 0.35:
        return dict(scene="field", quads=rng.randint(16, 256), spheres=rng.randint(1, 64))
    return dict(scene="soup", n=_log(rng, 300, n_hi))


def draw(rng):
    kind = rng.choice(["build", "build", "trace", "trace", "ao", "pt", "diff", "batch"])
    if kind == "build":
        builder = rng.choice(["lbvh", "lbvh", "ploc"])
        return dict(kind="build", builder=builder, normal=rng.random() < 0.25, **_draw_scene(rng))
    if kind == "trace":
        case = dict(kind="trace", form=rng.choice(["plain", "replay", "wide", "qwide", "quantised"]),
                    query=rng.choice(["closest", "any"]), **_draw_scene(rng))
        if rng.random() < 0.4:
            case.update(rays="camera", w=_log(rng, 64, 1920), h=_log(rng, 64, 1080))
        else:
            case.update(rays="random", nrays=_log(rng, 257, MAX_RAYS))
        return case
    if kind == "ao":
        return dict(kind="ao", form=rng.choice(["plain", "replay", "wide", "qwide", "quantised"]),
                    rebuild=rng.random() < 0.4, w=_log(rng, 64, 1280), h=_log(rng, 64, 720),
                    samples=_log(rng, 4, 64), radius=round(rng.uniform(0.05, 0.4), 3), sobol=rng.random() < 0.75,
                    **_draw_scene(rng, MAX_TRIS // 2))
    if kind == "pt":
        return dict(kind="pt", walk=rng.choice(["plain", "replay"]), w=_log(rng, 48, 1024), h=_log(rng, 48, 768),
                    sobol=rng.random() < 0.75, scene="field", quads=rng.randint(16, 256), spheres=rng.randint(1, 64))
    if kind == "diff":
        return dict(kind="diff", w=_log(rng, 32, 512), h=_log(rng, 32, 512), spp=_log(rng, 1, 64),
                    bounces=rng.randint(1, 3), quads=rng.randint(16, 256), spheres=rng.randint(1, 64))
    return dict(kind="batch", meshes=_log(rng, 2, 256), tri_lo=rng.randint(1, 64), tri_hi=_log(rng, 512, 65_536),
                ray_lo=rng.randint(64, 1024), ray_hi=_log(rng, 2048, 262_144), counts_seed=rng.randint(0, 10_000),
                query=rng.choice(["closest", "any"]))


# ------------------------------------------------------------------ the inputs
def _scene(case, seed):
    """The case's triangles, float32 (n, 9) on the GPU."""
    if case["scene"] == "field":
        t = scenes.heightfield_icospheres(seed % SEED_CAP, quads=case["quads"], spheres=case["spheres"])
        return torch.from_numpy(t).cuda()
    return scenes.batched_soup(1, case["n"], case["n"], seed % SEED_CAP, "cuda")[0]


def _count(case):
    """The case's triangles, as a number."""
    if case["kind"] == "batch":
        return int(_batch_counts(case)[0].sum())
    if "n" in case:
        return case["n"]
    return 2 * case["quads"] ** 2 + 1280 * case["spheres"] + (2 if case["kind"] == "diff" else 0)


def _camera(case):
    view = scenes.camera_soup() if case.get("scene") == "soup" else scenes.camera_heightfield()
    return mb.RayGenerator().lookat(*view, case["w"], case["h"])


def _ray_count(case):
    return case["nrays"] if case["rays"] == "random" else (case["w"] * case["h"] + 1) // 2


def _rays(case, tris, seed):
    if case["rays"] == "camera":
        c = _camera(case)
        rays = scenes.camera_rays(c.m_origin, c.m_right, c.m_up, case["w"], case["h"])
    else:
        p = tris.view(-1, 3)
        rays = scenes.random_rays(case["nrays"], p.amin(0).cpu().numpy(), p.amax(0).cpu().numpy(),
                                  (seed + 1) % SEED_CAP)
        if case["query"] == "any":
            rays[:, 7] = 0.25  # shadow rays end at their light
    return torch.from_numpy(rays).cuda()


def _batch_counts(case):
    tri = scenes.log_uniform_counts(case["meshes"], case["tri_lo"], case["tri_hi"], case["counts_seed"])
    ray = scenes.log_uniform_counts(case["meshes"], case["ray_lo"], case["ray_hi"], case["counts_seed"] + 1)
    return tri, ray


def _form(case, builder, tris):
    """What a program keeps beside the built tree for the case's form."""
    form = case.get("form", case.get("walk"))
    if form == "replay":
        return mb.leaf_triangles(builder, tris)
    if form == "wide":
        return mb.WideBVH.from_builder(builder, tris)
    if form == "qwide":
        return mb.WideBVH.from_builder(builder, tris).quantise()
    if form == "quantised":
        return mb.QuantisedBVH.from_builder(builder, tris)
    return None


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "batch":
        counts, ray_counts = _batch_counts(case)
        n = int(counts.sum())
        offsets = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
        tris = scenes.batched_soup(1, n, n, seed % SEED_CAP, "cuda")[0]
        rays, ray_offsets = scenes.batched_rays(tris, offsets, seed=(seed + 1) % SEED_CAP, counts=ray_counts)
        b = mb.BatchedBVH(tris, torch.from_numpy(offsets.astype(np.int32)).cuda(), case["meshes"])
        query = mb.RAY_QUERY_ANY if case["query"] == "any" else mb.RAY_QUERY_CLOSEST
        s["batch"] = b.set_rays(rays, torch.from_numpy(ray_offsets.astype(np.int32)).cuda(), query)
        return s
    if kind == "diff":
        field = scenes.heightfield_icospheres(seed % SEED_CAP, quads=case["quads"], spheres=case["spheres"])
        tris = torch.from_numpy(np.concatenate([field, scenes.quad_light()])).cuda()
    else:
        tris = _scene(case, seed)
    n = len(tris)
    s["tris"] = tris
    s["sorter"] = mb.OnesweepSort()
    s["builder"] = mb.BVHGPUBuilder()
    if kind == "build":
        return s
    b = s["builder"].build(tris, n, 0, s["sorter"])
    s["form"] = _form(case, b, tris)
    if kind == "trace":
        s["rays"] = _rays(case, tris, seed)
        s["hits"] = torch.empty((len(s["rays"]), 8), dtype=torch.int32, device="cuda")
        return s
    px = case["w"] * case["h"]
    s["camera"] = _camera(case)
    if kind == "ao":
        s["pixels"] = torch.zeros(px, dtype=torch.int32, device="cuda")
        s["occluded"] = torch.zeros(px, dtype=torch.int32, device="cuda")
    elif kind == "pt":
        s["attribs"] = torch.from_numpy(scenes.pt_attributes(n, (seed + 2) % SEED_CAP, 0.01)).cuda()
        s["accum"] = torch.zeros((px, 4), dtype=torch.float32, device="cuda")
        s["pixels"] = torch.zeros(px, dtype=torch.int32, device="cuda")
    else:
        s["albedo"] = torch.from_numpy(scenes.albedo(n, (seed + 3) % SEED_CAP)).cuda()
        s["emission"] = torch.zeros(n, dtype=torch.float32, device="cuda")
        s["emission"][-2:] = 10.0
        s["image"] = torch.zeros(px, dtype=torch.float32, device="cuda")
        s["target"] = torch.full((px,), 0.5, dtype=torch.float32, device="cuda")
        s["grad"] = torch.zeros(n, dtype=torch.float32, device="cuda")
    return s


# -------------------------------------------------------------------- the work
def _build(s):
    case, b, tris = s["case"], s["builder"], s["tris"]
    option = mb.BUILD_OPTION_USE_NORMAL if case.get("normal") else 0
    if case.get("builder") == "ploc":
        return b.buildByPLOC(tris, len(tris), option, s["sorter"])
    return b.build(tris, len(tris), option, s["sorter"])


def _trace(s):
    case, b, form = s["case"], s["builder"], s["form"]
    query = mb.RAY_QUERY_ANY if case["query"] == "any" else mb.RAY_QUERY_CLOSEST
    kind = case["form"]
    if kind in ("wide", "qwide"):
        return mb.intersect_wide(form, s["rays"], s["hits"], quantised=kind == "qwide", rayQuery=query)
    if kind == "quantised":
        return mb.intersect_quantised(form, s["rays"], query, s["hits"])
    if kind == "replay":
        return mb.intersect(b, s["tris"], s["rays"], query, mb.TRAVERSAL_REPLAY, s["hits"])
    return mb.intersect(b, s["tris"], s["rays"], query, hits=s["hits"])


def _ao(s):
    case, b, tris = s["case"], s["builder"], s["tris"]
    kind = case["form"]
    if case["rebuild"]:
        _build(s)
        if kind in ("wide", "qwide"):
            s["form"].update()
        elif kind == "quantised":
            s["form"] = mb.QuantisedBVH.from_builder(b, tris)
        elif kind == "replay":
            mb.leaf_triangles(b, tris, out=s["form"])
    size, args = (case["w"], case["h"]), (int(case["sobol"]), case["samples"], case["radius"], 12345)
    if kind in ("wide", "qwide"):
        mb.render_ao_wide(s["pixels"], size, s["camera"], s["form"], *args, occluded=s["occluded"],
                          quantised=kind == "qwide")
    elif kind == "quantised":
        mb.render_ao_quantised(s["pixels"], size, s["camera"], s["form"], *args, occluded=s["occluded"])
    elif kind == "replay":
        mb.render_ao(s["pixels"], size, s["camera"], b.m_rootNode, b.m_internals, tris, *args,
                     occluded=s["occluded"], traversal=mb.TRAVERSAL_REPLAY, leaf_triangles=s["form"])
    else:
        mb.render_ao(s["pixels"], size, s["camera"], b.m_rootNode, b.m_internals, tris, *args,
                     occluded=s["occluded"])
    return s["pixels"], s["occluded"]


def _pt(s):
    case, b = s["case"], s["builder"]
    size = (case["w"], case["h"])
    walk = mb.TRAVERSAL_REPLAY if case["walk"] == "replay" else mb.TRAVERSAL_STACKFREE
    mb.render_pt(s["accum"], size, s["camera"], b.m_rootNode, b.m_internals, s["tris"], s["attribs"],
                 int(case["sobol"]), traversal=walk, leaf_triangles=s["form"])
    mb.pack(s["pixels"], s["accum"], case["w"] * case["h"])
    return s["accum"], s["pixels"]


def _diff(s):
    case, b = s["case"], s["builder"]
    size, args = (case["w"], case["h"]), (s["tris"], s["albedo"], s["emission"], case["spp"], case["bounces"])
    mb.pt_diff_render(s["image"], size, s["camera"], b, *args)
    s["grad"].zero_()
    mb.pt_diff_adjoint(s["grad"], (s["image"] - s["target"]) * (2.0 / len(s["image"])), size, s["camera"], b, *args)
    return s["image"], s["grad"]


def run(state):
    kind = state["case"]["kind"]
    if kind == "build":
        b = _build(state)
        return b.nodes, b.m_rootNode[:1], b.m_sceneAABB[:6]
    if kind == "trace":
        return _trace(state)
    if kind == "ao":
        return _ao(state)
    if kind == "pt":
        return _pt(state)
    if kind == "diff":
        return _diff(state)
    b = state["batch"].build()
    hits = b.trace()
    return b.internals, b.roots[:b.nMeshes], b.mesh_aabbs, hits


# --------------------------------------------------------- what it cannot skip
def _ray_flops(n):
    """One descent to a leaf, two boxes a level, and one triangle test."""
    return 24 * max(1.0, math.log2(n)) + 70


def work(case):
    n = _count(case)
    kind = case["kind"]
    tree = 100 * n  # nodes and triangles
    if kind == "build":
        return {"bytes": 36 * n + 64 * (n - 1) + 28, "flops": 40 * n}
    if kind == "trace":
        r = _ray_count(case)
        return {"bytes": 64 * r + min(tree, 256 * r), "flops": r * _ray_flops(n)}
    px = case.get("w", 0) * case.get("h", 0)
    if kind == "ao":
        r = px * (1 + case["samples"])
        built = 164 * n if case["rebuild"] else 0
        return {"bytes": 8 * px + min(tree, 256 * r) + built, "flops": r * _ray_flops(n)}
    if kind == "pt":
        return {"bytes": 36 * px + min(tree, 512 * px), "flops": 3 * px * _ray_flops(n)}
    if kind == "diff":
        r = px * case["spp"] * (1 + case["bounces"])
        return {"bytes": 12 * px + 12 * n + min(tree, 256 * r), "flops": 2 * r * _ray_flops(n)}
    r = int(_batch_counts(case)[1].sum())
    return {"bytes": 36 * n + 64 * (n - case["meshes"]) + 64 * r + tree, "flops": 40 * n + r * _ray_flops(n)}


# ------------------------------------------------------------- in 64 bits
def exact(case, seed):
    """The bounds in 64 bits, where a build returns them (minima and maxima of the inputs); nodes and hits are words,
    which have to be equal, and the images' and gradients' paths take too long on the host."""
    if case["kind"] == "build":
        p = _scene(case, seed).double().view(-1, 3)
        return None, None, torch.cat([p.amin(0), p.amax(0)])
    if case["kind"] == "batch":
        counts, _ = _batch_counts(case)
        n = int(counts.sum())
        p = scenes.batched_soup(1, n, n, seed % SEED_CAP, "cuda")[0].double().view(-1, 3, 3)
        parts = torch.split(p, counts.tolist())
        return None, None, torch.stack([torch.cat([q.amin((0, 1)), q.amax((0, 1))]) for q in parts]), None
    return None
