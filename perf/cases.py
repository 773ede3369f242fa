"""The work a user of this framework has it do, as cases that can be timed one by one.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare(case, seed)``
makes what a user's program has in hand before the call, ``run(state)`` is one call (or the calls of
one frame) through the public entry points, ``work(case)`` is what it cannot do without, and
``exact(case, seed)`` is the 64-bit value where there is one.

Four kinds of work:

* ``render``: passes of one progressive render and its image (``Renderer``),
* ``batch``: passes of many jobs in one set of launches and their images (``Batch``),
* ``hash`` and ``reduce``: the stage-level entry points on a caller's device arrays,
* ``bvh``: a mesh's threaded BVH built on the GPU.

A render goes on from where the last call left it, as a user's does.  The scene is the case's; the
seed draws the camera's place, the random sequence and every array that a stage entry point is given.
"""
from __future__ import annotations

import ctypes
import functools

import numpy as np
import torch

import glslppm_gb300 as g
from glslppm_gb300 import native, renderer, scenes

REDUCE_OPS = {"min": renderer.REDUCE_MIN, "max": renderer.REDUCE_MAX, "sum": renderer.REDUCE_SUM}


def _render(name, scene, detail, width, height, photon_width, photon_height, passes, *, precision="fp32",
            grid=False, hash_slots=0, radius="diagonal", eye_interval=10, image="radiance"):
    c = {"kind": "render", "scene": scene, "detail": detail, "width": width, "height": height,
         "photon_width": photon_width, "photon_height": photon_height, "passes": passes, "precision": precision,
         "grid": grid, "hash_slots": hash_slots, "radius": radius, "eye_interval": eye_interval, "image": image}
    return {"name": name, **c} if name else c


def _batch(name, jobs, first, max_tris, passes, *, precision="fp32", trim=0):
    c = {"kind": "batch", "jobs": jobs, "first": first, "max_tris": max_tris, "passes": passes,
         "precision": precision, "trim": trim}
    return {"name": name, **c} if name else c


def listed():
    return [
        # an interactive viewer's loop: a small window, one pass per frame, the displayed image read back
        _render("preview-128", "box", 64, 128, 128, 128, 128, 1, radius="footprint", image="display"),
        # the 256x256 workload, whole: 64 passes of 2^16 photons, then its image
        _render("box-256", "box", 64, 256, 256, 256, 256, 64),
        # the 1024x1024 workload: an eye-pass cycle of ten passes between image updates, in the plain
        # precision, the mixed one, and the mixed one with every photon gathered
        _render("box-1024", "box", 64, 1024, 1024, 1024, 1024, 10),
        _render("box-1024-mixed", "box", 64, 1024, 1024, 1024, 1024, 10, precision="mixed"),
        _render("box-1024-grid", "box", 64, 1024, 1024, 1024, 1024, 10, precision="mixed", grid=True),
        # every material class (glass, plastic, glossy) at sizes that divide nothing, the reference's
        # radius rule, a hash table larger than the photon buffer
        _render("materials-odd", "materials", 40, 603, 401, 517, 389, 20, radius="footprint", hash_slots=300007),
        # a mesh whose nodes and triangles do not fit in L2, at full HD with 2^21 photons
        _render("mesh-1m", "mesh", 512, 1920, 1080, 2048, 1024, 10),
        _render("mesh-1m-mixed", "mesh", 512, 1920, 1080, 2048, 1024, 10, precision="mixed"),
        # a render farm's batch: jobs of uneven triangle count, image size and photon budget
        _batch("batch-16", 16, 0, 100_000, 10),
        # the photon hash on a caller's arrays, one pass of the 1024x1024 workload's photons
        {"name": "hash-1024", "kind": "hash", "photon_width": 1024, "photon_height": 1024, "hash_slots": 1 << 20,
         "clip": True},
        # the reference's ReduceTexture on a caller's 1024x1024 texture
        {"name": "reduce-1024", "kind": "reduce", "resolution": 1024, "op": "sum"},
        # the threaded BVH of a loaded mesh, before its first upload
        {"name": "bvh-260k", "kind": "bvh", "detail": 256},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "render", "batch", "hash", "reduce", "bvh"])
    if kind == "render":
        scene = rng.choice(["box", "box", "materials", "environment", "mesh"])
        detail = _log(rng, 32, 400) if scene == "mesh" else 2 * _log(rng, 6, 48)
        precision = rng.choice(["fp32", "fp32", "mixed"])
        w, h = _log(rng, 48, 1400), _log(rng, 48, 1000)
        pw, ph = _log(rng, 48, 1400), _log(rng, 48, 1000)
        cost = w * h + 2 * pw * ph  # of one pass, against the largest listed render's ten
        passes = max(1, min(_log(rng, 1, 40), int(3e7 / cost)))
        return _render(None, scene, detail, w, h, pw, ph, passes, precision=precision,
                       grid=precision == "mixed" and rng.random() < 0.4,
                       hash_slots=rng.choice([0, 0, 2 * pw * ph + 1]), radius=rng.choice(["diagonal", "footprint"]),
                       eye_interval=rng.choice([1, 4, 10, 10]), image=rng.choice(["radiance", "display"]))
    if kind == "batch":
        return _batch(None, rng.randint(2, 16), rng.randint(0, 200), _log(rng, 12_000, 60_000), rng.randint(1, 10),
                      precision=rng.choice(["fp32", "mixed"]), trim=rng.choice([0, 5, 27]))
    if kind == "hash":
        w, h = _log(rng, 64, 2048), _log(rng, 64, 1024)
        return {"kind": "hash", "photon_width": w, "photon_height": h,
                "hash_slots": rng.choice([w * h, 2 * w * h + 1, max(w * h // 2, 1)]), "clip": rng.random() < 0.5}
    if kind == "reduce":
        return {"kind": "reduce", "resolution": 1 << rng.randint(2, 13), "op": rng.choice(["min", "max", "sum"])}
    return {"kind": "bvh", "detail": _log(rng, 40, 300)}


# ---- scenes ------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _mesh(scene, detail):
    """A case's scene with its BVH: built once in a program that renders it."""
    if scene == "box":
        return scenes.cornell_box(detail, detail // 2).to_mesh()
    if scene in ("materials", "environment"):
        return scenes.materials_box(detail, detail // 2, light=scene == "materials").to_mesh()
    s = scenes.large_mesh(1, sphere_freq=max(4, round(detail * 0.309)), floor_verts=detail)
    return g.Mesh.from_arrays(s.positions, s.material_ids, s.material_array(), s.normals).build_bvh(gpu=True)


@functools.lru_cache(maxsize=64)
def _variant(seed, max_tris):
    """A batch job's sizes and its scene, prepared once as a server that renders it often does."""
    s = scenes.cornell_variant(seed, min(10_000, max_tris), max_tris)
    m = g.Mesh.from_arrays(s.scene.positions, s.scene.material_ids, s.scene.material_array(), s.scene.normals)
    return (s.width, s.height, s.photon_width, s.photon_height), g.PreparedScene(m.build_bvh(gpu=True))


def _camera(scene, width, height, rng):
    """A camera near the scene's own, moved and turned a little by the seed."""
    origin, lookat = ((0.0, 1.6, 3.2), (0.0, 0.6, 0.0)) if scene == "mesh" else ((0.5, 0.5, 2.15), (0.5, 0.5, 0.0))
    o = np.asarray(origin) + rng.uniform(-0.06, 0.06, 3)
    a = np.asarray(lookat) + rng.uniform(-0.06, 0.06, 3)
    return g.look_at(tuple(map(float, o)), tuple(map(float, a)), width, height)


def _config(case, width, height, photon_width, photon_height, seed):
    mixed = case["precision"] == "mixed"
    diagonal = case.get("radius", "diagonal") == "diagonal"
    return g.default_config(width, height=height, photon_width=photon_width, photon_height=photon_height,
                            hash_slots=case.get("hash_slots", 0),
                            radius_rule=native.RADIUS_DIAGONAL if diagonal else native.RADIUS_FOOTPRINT,
                            radius_fraction=0.005, eye_pass_interval=case.get("eye_interval", 10), seed=seed,
                            precision=native.PRECISION_MIXED if mixed else native.PRECISION_FP32,
                            flags=native.FLAG_PHOTON_GRID if case.get("grid") else 0)


# ---- what a program has in hand, and one call ----------------------------------------------------------------------
def prepare(case, seed):
    rng = np.random.default_rng([int(seed), 0x5eed])
    return {"render": _prepare_render, "batch": _prepare_batch, "hash": _prepare_hash, "reduce": _prepare_reduce,
            "bvh": _prepare_bvh}[case["kind"]](case, rng)


def run(state):
    return {"render": _run_render, "batch": _run_batch, "hash": _run_hash, "reduce": _run_reduce,
            "bvh": _run_bvh}[state["kind"]](state)


def _prepare_render(case, rng):
    w, h = case["width"], case["height"]
    r = g.Renderer(_config(case, w, h, case["photon_width"], case["photon_height"], int(rng.integers(1, 1 << 31))))
    r.upload_scene(_mesh(case["scene"], case["detail"]))
    cam = _camera(case["scene"], w, h, rng)
    r.set_camera(cam)
    r.synchronize()
    kind = native.IMAGE_DISPLAY if case["image"] == "display" else native.IMAGE_RADIANCE
    return {"kind": "render", "renderer": r, "camera": cam, "passes": case["passes"], "image_kind": kind,
            "image": g.pinned_empty((h, w, 3))}


def _run_render(state):
    r = state["renderer"]
    r.run_passes(state["passes"])
    return r.read_image(state["image_kind"], state["image"])


def _prepare_batch(case, rng):
    jobs = [_variant(case["first"] + k, case["max_tris"]) for k in range(case["jobs"])]
    mixed = case["precision"] == "mixed"
    b = g.Batch(precision=native.PRECISION_MIXED if mixed else native.PRECISION_FP32, max_jobs=len(jobs))
    ids, images = [], []
    for (w, h, pw, ph), scene in jobs:
        w, h = w - case["trim"], h - case["trim"]
        cfg = _config(case, w, h, pw, ph, int(rng.integers(1, 1 << 31)))
        ids.append(b.add_job_prepared(cfg, scene, _camera("box", w, h, rng)))
        images.append(g.pinned_empty((h, w, 3)))
    b.synchronize()
    return {"kind": "batch", "batch": b, "ids": ids, "images": images, "passes": case["passes"]}


def _run_batch(state):
    b = state["batch"]
    b.run_passes(state["passes"])
    for job, image in zip(state["ids"], state["images"]):
        b.read_image_async(job, image)
    b.synchronize()
    return state["images"]


def _prepare_hash(case, rng):
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1, 1 << 31)))
    n = case["photon_width"] * case["photon_height"]
    # photons on the faces of a unit box, a few of them bunched (a caustic); a quarter is not stored
    pos = torch.rand((n, 4), generator=gen, device="cuda")
    face = torch.randint(0, 3, (n, 1), generator=gen, device="cuda")
    pos.scatter_(1, face, torch.round(pos.gather(1, face)))
    bunched = torch.rand((n, 1), generator=gen, device="cuda") < 0.05
    pos = torch.where(bunched, 0.3 + 0.02 * pos, pos).contiguous()
    flux = torch.rand((n, 4), generator=gen, device="cuda")
    flux[torch.rand(n, generator=gen, device="cuda") < 0.25] = -1.0
    slots = case["hash_slots"]
    return {"kind": "hash", "pos": pos, "flux": flux, "case": case,
            "winner": torch.empty(slots, dtype=torch.int32, device="cuda"),
            "count": torch.empty(slots, dtype=torch.int32, device="cuda")}


def _run_hash(state):
    c = state["case"]
    renderer.hash_build(state["pos"].data_ptr(), state["flux"].data_ptr(), c["photon_width"], c["photon_height"],
                        c["hash_slots"], (-0.01, -0.01, -0.01), 57.7, native.FLAG_GL_DEPTH_CLIP if c["clip"] else 0,
                        state["winner"].data_ptr(), state["count"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return {"winner": state["winner"], "count": state["count"]}


def _texture(case, rng):
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1, 1 << 31)))
    n = case["resolution"]
    # hit positions with a coverage count in w, as the reference reduces them
    t = torch.rand((n, n, 4), generator=gen, device="cuda") * 2.0
    t[..., 3] = (t[..., 3] > 0.6).float()
    return t


def _prepare_reduce(case, rng):
    return {"kind": "reduce", "texture": _texture(case, rng), "resolution": case["resolution"],
            "op": REDUCE_OPS[case["op"]]}


def _run_reduce(state):
    return renderer.reduce_texture(state["texture"].data_ptr(), state["resolution"], state["op"],
                                   torch.cuda.current_stream().cuda_stream)


def _prepare_bvh(case, rng):
    d = case["detail"]
    seed = int(rng.integers(1, 1 << 20))
    geo = np.concatenate([scenes.geodesic_sphere((0.0, 0.75, 0.0), 0.6, max(4, round(d * 0.309)), 0.08, seed),
                          scenes.heightfield(2.0, d, 0.1, seed)]).astype(np.float32)
    mats = np.zeros(1, dtype=renderer.MATERIAL_DTYPE)
    mats[0]["color"], mats[0]["eta"] = (0.7, 0.7, 0.7), 1.7
    return {"kind": "bvh", "mesh": g.Mesh.from_arrays(geo, np.zeros(len(geo), np.int32), mats)}


def _view(owner, pointer, ctype, shape):
    """A numpy view of an array that `owner` holds, and that keeps the owner alive."""
    buf = (ctype * int(np.prod(shape))).from_address(ctypes.cast(pointer, ctypes.c_void_p).value)
    buf._owner = owner
    return np.frombuffer(buf, dtype=ctype).reshape(shape)


def _run_bvh(state):
    mesh = state["mesh"].build_bvh(gpu=True)
    s = mesh.scene()
    n = s.num_nodes
    return {"node_bounds": _view(mesh, s.node_bounds, ctypes.c_float, (n, 6)),
            "node_triangle": _view(mesh, s.node_triangle, ctypes.c_int32, (n,)),
            "order_base": _view(mesh, s.order_base, ctypes.c_int32, (6, n)),
            "order_miss": _view(mesh, s.order_miss, ctypes.c_int32, (6, n))}


# ---- what a call cannot do without ---------------------------------------------------------------------------------
# One pass of a render reads and writes each photon's record (position, flux, direction, random state and
# the hit before: 72 bytes), reads each pixel's hit point (52) and reads and writes its statistics (32),
# and writes each hash slot's winner and count (8); the image is 12 bytes a pixel.  The arithmetic is a
# photon's: about 26 boxes of 20 operations, two triangles of 60, and its generation and storing.
def _pass_work(pixels, photons, slots):
    return 144 * photons + 116 * pixels + 8 * slots, 1000 * photons + 200 * pixels


def work(case):
    kind = case["kind"]
    if kind == "render":
        pixels, photons = case["width"] * case["height"], case["photon_width"] * case["photon_height"]
        b, f = _pass_work(pixels, photons, case["hash_slots"] or photons)
        return {"bytes": case["passes"] * b + 12 * pixels, "flops": case["passes"] * f}
    if kind == "batch":
        total_b = total_f = 0
        for k in range(case["jobs"]):
            (w, h, pw, ph), _ = _variant(case["first"] + k, case["max_tris"])
            w, h = w - case["trim"], h - case["trim"]
            b, f = _pass_work(w * h, pw * ph, pw * ph)
            total_b += case["passes"] * b + 12 * w * h
            total_f += case["passes"] * f
        return {"bytes": total_b, "flops": total_f}
    if kind == "hash":
        n = case["photon_width"] * case["photon_height"]
        return {"bytes": 32 * n + 8 * case["hash_slots"], "flops": 60 * n}
    if kind == "reduce":
        n = case["resolution"] ** 2
        return {"bytes": 16 * n + 16, "flops": 4 * n}
    d = case["detail"]
    tris = 20 * max(4, round(d * 0.309)) ** 2 + 2 * (d - 1) ** 2
    # the triangles' vertices in; a node's box, triangle and its base and miss link in six orderings out
    return {"bytes": 36 * tris + 2 * tris * (24 + 4 + 48), "flops": 2 * tris * 400}


def exact(case, seed):
    """The reduction in 64 bits.  The hash and the BVH's links are whole numbers, and a render draws its
    random sequence in single precision by its definition: those have no other value to be held to."""
    if case["kind"] != "reduce":
        return None
    t = _texture(case, np.random.default_rng([int(seed), 0x5eed])).double().reshape(-1, 4)
    v = {"min": lambda: t.amin(0), "max": lambda: t.amax(0), "sum": lambda: t.sum(0)}[case["op"]]()
    return v.cpu().numpy()
