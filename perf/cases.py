"""The work that programs built on obvh_b200 have it do, as measurable cases.

``listed()`` names twelve cases, ``draw(rng)`` makes one more of the same
ranges, ``prepare(case, seed)`` makes what a program holds before the call,
``run(state)`` is one pass through the public entry points, ``work(case)`` the
bytes and operations that a pass cannot do without and ``exact(case, seed)``
the outputs in 64 bits where they are computed numbers that do not hang on a
choice rounded in 32 bits (a tree's topology is such a choice).

Kinds:

* ``fit``        one point set already on the device (DitoFitter.fit)
* ``fit_host``   one point set in host memory (kr_cuda_points_obb)
* ``fit_batch``  many point sets of uneven sizes (DitoBatch)
* ``build``      LBVH, with the OBB tree and the collapse as asked (ObvhBuilder)
* ``atrbvh``     the same commit with the treelet-optimised tree (AtrbvhBuilder)
* ``build_batch`` many meshes of uneven sizes in one launch (BuildBatch)
* ``transform``  the OBB tree of a tree that exists (kr_cuda_bvh_obb_tree)
* ``pack``       the traversal layouts of a collapsed OBB tree (obvh_pack)
* ``trace``      closest hits of rays through the packed tree (soa_obvh_intersect)
"""
import math

import numpy as np
import torch

from obvh_b200 import REFERENCE_GPU, DitoFitter, bvh, kr_cuda_points_obb, workloads
from obvh_b200.batch import DitoBatch

DEV = "cuda"


def listed():
    return [
        # the box of one small object (a prop, a bone's skin) that lies on the device: a call whose latency counts
        {"name": "fit_4k", "kind": "fit", "cloud": "gaussian", "points": 4093, "gpu_rules": False},
        # the reference's own call: an object's vertices in host memory, the box by value
        {"name": "fit_host_100k", "kind": "fit_host", "points": 100003},
        # a laser scan: the largest single set that the benchmark fits
        {"name": "fit_100m", "kind": "fit", "cloud": "ellipsoid", "points": 100_000_000, "gpu_rules": False},
        # the boxes of every object of a scene at once, 64 to 262,144 points each
        {"name": "fit_batch_4096", "kind": "fit_batch", "sets": 4096, "smallest": 64, "largest": 262144, "layout": 3},
        # one small mesh committed by itself: a chain of launches over next to no data
        {"name": "build_1k", "kind": "build", "mesh": "soup", "triangles": 1021, "obbs": True, "collapse": True,
         "ci": 1.2, "replay": False},
        # a hairball-like scene of two million triangles rebuilt in place every frame from a captured graph
        {"name": "build_2m_replay", "kind": "build", "mesh": "soup", "triangles": 2_000_000, "obbs": True,
         "collapse": True, "ci": 1.2, "replay": True},
        # a closed mesh committed with the optimised tree, which pays for itself over many rays
        {"name": "atrbvh_917k", "kind": "atrbvh", "segments": 1024, "around": 448, "treelet": 9, "obbs": True,
         "collapse": True},
        # every mesh of a scene committed in one launch, 64 to 16,384 triangles each
        {"name": "build_batch_2048", "kind": "build_batch", "meshes": 2048, "smallest": 64, "largest": 16384,
         "layout": 5},
        # a tree that another builder made, turned into an OBB tree by the reference's call
        {"name": "transform_230k", "kind": "transform", "segments": 513, "around": 224},
        # the layouts for traversal, made after each commit of the large scene
        {"name": "pack_2m", "kind": "pack", "triangles": 2_000_000},
        # a bounce of a path tracer: rays from anywhere to anywhere
        {"name": "trace_probe_2m", "kind": "trace", "mesh": "soup", "triangles": 2_000_000, "rays": 2_000_003,
         "camera": False},
        # the first rays of a picture, 1920 x 1080, neighbours almost alike
        {"name": "trace_camera_1080p", "kind": "trace", "mesh": "knot", "segments": 1024, "around": 448,
         "rays": 1920 * 1080, "camera": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit_host", "fit_batch", "build", "build", "build", "atrbvh", "atrbvh",
                       "build_batch", "transform", "pack", "trace", "trace"])
    c = {"kind": kind}
    if kind == "fit":
        c.update(cloud=rng.choice(["gaussian", "ellipsoid"]), points=_log(rng, 64, 60_000_000),
                 gpu_rules=rng.random() < 0.2)
    elif kind == "fit_host":
        c.update(points=_log(rng, 1000, 100_003))
    elif kind == "fit_batch":
        c.update(sets=_log(rng, 64, 4000), smallest=64, largest=_log(rng, 4096, 262144), layout=rng.randrange(1 << 20))
    elif kind == "build":
        flags = rng.choice([(True, True), (True, True), (True, False), (False, True), (False, False)])
        if rng.random() < 0.7:
            c.update(mesh="soup", triangles=_log(rng, 1021, 2_000_000))
        else:
            c.update(mesh="knot", segments=_log(rng, 32, 1024), around=_log(rng, 16, 448))
        c.update(obbs=flags[0], collapse=flags[1], ci=rng.choice([1.2, 1.2, 2.0, 0.8]), replay=rng.random() < 0.5)
    elif kind == "atrbvh":
        c.update(segments=_log(rng, 64, 1024), around=_log(rng, 32, 448), treelet=rng.choice([7, 9, 9]), obbs=True,
                 collapse=rng.random() < 0.8)
    elif kind == "build_batch":
        c.update(meshes=_log(rng, 32, 2000), smallest=64, largest=_log(rng, 1024, 16384), layout=rng.randrange(1 << 20))
    elif kind == "transform":
        c.update(segments=_log(rng, 64, 512), around=_log(rng, 32, 224))
    elif kind == "pack":
        c.update(triangles=_log(rng, 1021, 2_000_000))
    else:
        c.update(camera=rng.random() < 0.5, rays=_log(rng, 4093, 2_000_000))
        if rng.random() < 0.5:
            c.update(mesh="soup", triangles=_log(rng, 10_007, 2_000_000))
        else:
            c.update(mesh="knot", segments=_log(rng, 64, 1024), around=_log(rng, 32, 448))
    return c


# ---- inputs ---------------------------------------------------------------------
def _points(case, seed):
    if case.get("cloud") == "ellipsoid":
        return workloads.ellipsoid_points_torch(case["points"], seed=seed, device=DEV)
    return workloads.gaussian_cloud_torch(case["points"], np.random.default_rng(seed), device=DEV)


def _sizes(count, smallest, largest, layout):
    rng = np.random.default_rng(layout)
    sizes = np.exp(rng.uniform(math.log(smallest), math.log(largest), size=count)).astype(np.int64)
    offsets = np.zeros(count + 1, np.int64)
    np.cumsum(sizes, out=offsets[1:])
    return sizes, offsets


def _cloud_sets(case, seed):
    """Anisotropic Gaussian clouds (per-axis sigma log-uniform, turned and moved) in one packed array."""
    sizes, offsets = _sizes(case["sets"], case["smallest"], case["largest"], case["layout"])
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    s = case["sets"]
    q = torch.randn((s, 4), generator=g, device=DEV, dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                       2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                       2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).reshape(s, 3, 3)
    sigma = torch.exp(torch.empty((s, 1, 3), device=DEV, dtype=torch.float64).uniform_(math.log(0.01), math.log(5.0),
                                                                                       generator=g))
    frame = (rot * sigma).to(torch.float32)
    move = torch.empty((s, 3), device=DEV).uniform_(-100.0, 100.0, generator=g)
    out = torch.empty((int(offsets[-1]), 3), dtype=torch.float32, device=DEV)
    for a in range(0, s, 512):
        b = min(s, a + 512)
        lo, hi = int(offsets[a]), int(offsets[b])
        of = torch.repeat_interleave(torch.arange(a, b, device=DEV), torch.from_numpy(sizes[a:b]).to(DEV))
        p = torch.randn((hi - lo, 3), generator=g, device=DEV)
        for k in range(3):
            out[lo:hi, k] = (p * frame[of, k]).sum(1) + move[of, k]
    return out, offsets


def _mesh(case, seed):
    if case.get("mesh", "knot") == "soup":
        return bvh.Mesh.from_device(*workloads.triangle_soup_torch(case["triangles"], seed=seed, device=DEV))
    v, f = workloads.torus_knot_mesh(case["segments"], case["around"], seed=seed)
    return bvh.Mesh(v, f, device=DEV)


def _triangles(case):
    return case["triangles"] if "triangles" in case else 2 * case["segments"] * case["around"]


def _flags(case):
    return (bvh.BUILD_OBBS if case["obbs"] else 0) | (bvh.BUILD_COLLAPSE if case["collapse"] else 0)


def _rays(case, mesh, seed):
    """kr_ray records (origin, tmin, direction, tmax): either from the sphere around the mesh to points in its box, or
    a pinhole camera's, row by row, from a place on that sphere."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 77)
    lo, hi = mesh.verts.amin(0), mesh.verts.amax(0)
    centre, size = 0.5 * (lo + hi), (hi - lo).norm()
    n = case["rays"]
    r = torch.zeros((n, 8), dtype=torch.float32, device=DEV)
    if case["camera"]:
        eye = torch.randn(3, generator=g, device=DEV)
        eye = centre + size * eye / eye.norm()
        forward = (centre - eye) / size
        up = torch.tensor([0.0, 0.0, 1.0], device=DEV) if abs(float(forward[2])) < 0.9 else torch.tensor([0.0, 1.0, 0.0], device=DEV)
        right = torch.linalg.cross(forward, up)
        right = right / right.norm()
        up = torch.linalg.cross(right, forward)
        width = max(1, int(round(math.sqrt(n * 16 / 9))))
        i = torch.arange(n, device=DEV)
        x = ((i % width).float() + 0.5) / width - 0.5
        y = ((i // width).float() + 0.5) / (n / width) - 0.5
        r[:, 0:3] = eye
        r[:, 4:7] = forward + 1.2 * x[:, None] * right - 0.675 * y[:, None] * up
    else:
        u = torch.randn((n, 3), generator=g, device=DEV)
        o = centre + size * u / u.norm(dim=1, keepdim=True)
        r[:, 0:3] = o
        r[:, 4:7] = lo + torch.rand((n, 3), generator=g, device=DEV) * (hi - lo) - o
    r[:, 7] = 1e30
    return r.view(torch.uint8).reshape(-1)


def _built(builder, mesh):
    out = builder.build(mesh)
    err = builder.status(mesh.n_faces)[0]
    if err:
        raise RuntimeError("the build reported device error %d" % err)
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "fit":
        s.update(points=_points(case, seed), fitter=DitoFitter(DEV), out=torch.empty(15, device=DEV),
                 flags=REFERENCE_GPU if case["gpu_rules"] else 0)
    elif kind == "fit_host":
        s.update(points=_points(case, seed).cpu().numpy())
    elif kind == "fit_batch":
        points, offsets = _cloud_sets(case, seed)
        s.update(points=points, batch=DitoBatch(offsets), out=torch.empty((case["sets"], 15), device=DEV))
    elif kind in ("build", "atrbvh"):
        mesh = _mesh(case, seed)
        b = bvh.ObvhBuilder(DEV) if kind == "build" else bvh.AtrbvhBuilder(DEV)
        out = b.outputs(mesh.n_faces)
        keep = ["nodes", "parents", "counts", "costs", "bounds"]
        keep += ["obbs", "transforms"] if case["obbs"] else []
        keep += ["collapsed", "primitives"] if case["collapse"] else []
        args = {"flags": _flags(case), "ci": case.get("ci", 1.2)}
        if kind == "atrbvh":
            args["treelet_size"] = case["treelet"]
        s.update(mesh=mesh, builder=b, out=out, keep=keep, args=args,
                 graph=b.capture(mesh, out, **args) if case.get("replay") else None)
    elif kind == "build_batch":
        sizes, fo = _sizes(case["meshes"], case["smallest"], case["largest"], case["layout"])
        verts, faces = workloads.triangle_soup_torch(int(fo[-1]), seed=seed, device=DEV)
        first = torch.repeat_interleave(torch.from_numpy(3 * fo[:-1]).to(DEV), torch.from_numpy(sizes).to(DEV))
        faces[:, :3] -= first[:, None].to(faces.dtype)
        b = bvh.BuildBatch(3 * fo, fo, device=DEV)
        out = b.outputs()
        b.capture(verts, faces, out)
        s.update(verts=verts, faces=faces, batch=b, out=out)
    elif kind == "transform":
        mesh = _mesh(case, seed)
        b = bvh.AtrbvhBuilder(DEV)
        tree = b.build(mesh, flags=0)
        nn = 2 * mesh.n_faces - 1
        s.update(mesh=mesh, tree=tree, obbs=torch.empty((nn, 15), device=DEV), xfs=torch.empty((nn, 16), device=DEV))
    elif kind == "pack":
        n = case["triangles"]
        o = _built(bvh.ObvhBuilder(DEV), _mesh({"mesh": "soup", "triangles": n}, seed))
        s.update(nodes=o["collapsed"], xfs=o["transforms"], n=n,
                 packed=torch.zeros((2 * n - 1) * 64, dtype=torch.uint8, device=DEV),
                 pairs=torch.zeros(max(n - 1, 1) * 32, device=DEV))
    else:
        mesh = _mesh(case, seed)
        n = mesh.n_faces
        o = _built(bvh.ObvhBuilder(DEV), mesh)
        soa = bvh.obvh_pack(o["collapsed"], 2 * n - 1, n - 1, o["transforms"])
        s.update(mesh=mesh, n=n, prims=o["primitives"], rays=_rays(case, mesh, seed),
                 soa={k: soa[k] for k in ("left_T", "right_T", "metadata")},
                 isects=torch.empty(case["rays"] * 28, dtype=torch.uint8, device=DEV))
    torch.cuda.synchronize()
    return s


# ---- one pass ---------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "fit":
        return s["fitter"].fit(s["points"], out=s["out"], flags=s["flags"])
    if kind == "fit_host":
        return kr_cuda_points_obb(s["points"])[0]
    if kind == "fit_batch":
        s["batch"].run(s["points"], s["out"])
        return s["out"]
    if kind in ("build", "atrbvh"):
        if s["graph"] is not None:
            s["graph"].launch()
        else:
            s["builder"].build(s["mesh"], out=s["out"], **s["args"])
        return {k: s["out"][k] for k in s["keep"]}
    if kind == "build_batch":
        s["batch"].launch()
        return s["out"]
    if kind == "transform":
        return list(bvh.obb_tree(s["mesh"], s["tree"], s["obbs"], s["xfs"]))
    if kind == "pack":
        n = s["n"]
        return bvh.obvh_pack(s["nodes"], 2 * n - 1, n - 1, s["xfs"], packed=s["packed"], pairs=s["pairs"])
    isects, err = bvh.soa_obvh_intersect(s["soa"], s["mesh"], s["prims"], s["rays"], 2 * s["n"] - 1, s["n"] - 1,
                                         isects=s["isects"])
    return {"isects": isects, "error": err}


# ---- what a pass cannot do without ----------------------------------------------------
def _tree_work(n, vertices, obbs, collapse, trees=1):
    """Bytes: the mesh read, every output record written.  Operations, with OBBs: per internal node 37 projections of
    14 points (5 operations each), and each triangle's three vertices on three axes in each of its ancestors."""
    nn = 2 * n - trees
    size = 12 * vertices + 16 * n + nn * (36 + 12)
    size += nn * 124 if obbs else 0
    size += nn * 36 + 4 * n if collapse else 0
    ops = 0.0
    if obbs:
        ops = max(n - trees, 0) * 37 * 14 * 5 + n * math.log2(max(n / trees, 2)) * 45
    return {"bytes": float(size), "flops": float(ops)}


def _vertices(case):
    return 3 * case["triangles"] if "triangles" in case else case["segments"] * case["around"]


def work(case):
    kind = case["kind"]
    if kind in ("fit", "fit_host"):
        # each point once; 11 additions and 14 comparisons for the slabs, 15 operations and 6 comparisons for the box
        return {"bytes": 12.0 * case["points"] + 60, "flops": 46.0 * case["points"]}
    if kind == "fit_batch":
        n = int(_sizes(case["sets"], case["smallest"], case["largest"], case["layout"])[1][-1])
        return {"bytes": 12.0 * n + 60.0 * case["sets"], "flops": 46.0 * n}
    if kind in ("build", "atrbvh"):
        return _tree_work(_triangles(case), _vertices(case), case["obbs"], case["collapse"])
    if kind == "build_batch":
        n = int(_sizes(case["meshes"], case["smallest"], case["largest"], case["layout"])[1][-1])
        return _tree_work(n, 3 * n, True, True, case["meshes"])
    if kind == "transform":
        n = _triangles(case)
        w = _tree_work(n, _vertices(case), True, False)
        return {"bytes": w["bytes"] - 8.0 * (2 * n - 1), "flops": w["flops"]}  # nodes and parents read, boxes written
    n = _triangles(case)
    if kind == "pack":
        # per node its record read, its packed record and metadata written; per internal node the children's
        # transforms read, the pair and two 4x3 rows written
        return {"bytes": float((2 * n - 1) * (36 + 64 + 16) + (n - 1) * (128 + 128 + 96)), "flops": 0.0}
    # rays read and records written; of the tree and the mesh no more than the rays can touch (about 60 nodes each)
    tree = (n - 1) * 96 + (2 * n - 1) * 16 + 12 * _vertices(case) + 20 * n
    rays = case["rays"]
    return {"bytes": 60.0 * rays + min(float(tree), 7200.0 * rays), "flops": rays * 60.0 * 2 * 48}


# ---- the fits in 64 bits ----------------------------------------------------------------
def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


def _area(d):
    return d[..., 0] * d[..., 1] + d[..., 0] * d[..., 2] + d[..., 1] * d[..., 2]


def _box64(points, gpu_rules=False):
    """The DiTO-14 box [15] of one set of more than 14 points in general position."""
    coords = [points[:, k].double() for k in range(3)]
    sel, span = [None] * 14, [None] * 14
    for k, (a, b, c) in enumerate([(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1), (1, 1, -1), (1, -1, 1), (1, -1, -1)]):
        v = a * coords[0] + b * coords[1] + c * coords[2]
        for j, e in ((k, v.amin()), (7 + k, v.amax())):
            sel[j], span[j] = points[torch.nonzero(v == e)[0, 0]].double(), e
    sel, span = torch.stack(sel), torch.stack(span)
    lo, hi = span[0:3], span[7:10]
    far = (sel[:7] - sel[7:]).norm(dim=1).argmax()
    p0, p1 = sel[far], sel[far + 7]
    e0 = _unit(p0 - p1)
    u = sel - p0
    p2 = sel[(_dot(u, u) - _dot(u, e0) ** 2).argmax()]
    e1, e2 = _unit(p1 - p2), _unit(p2 - p0)
    base = _unit(torch.linalg.cross(e1, e0))
    t, level = _dot(sel, base), _dot(p0, base)
    frames = [(base, e0), (base, e1), (base, e2)]
    for apex, real in ((sel[t.argmax()], t.amax() - 1e-6 > level), (sel[t.argmin()], t.amin() + 1e-6 < level)):
        if real:
            f0, f1, f2 = _unit(apex - p0), _unit(apex - p1), _unit(apex - p2)
            for n, edges in ((torch.linalg.cross(f1, e0), (e0, f1, f0)), (torch.linalg.cross(f2, e1), (e1, f2, f1)),
                             (torch.linalg.cross(f0, e2), (e2, f0, f2))):
                frames += [(_unit(n), e) for e in edges]
    axes = torch.stack([torch.stack([e, n, torch.linalg.cross(e, n)]) for n, e in frames])  # [frames, 3, 3]
    proj = torch.einsum("fak,pk->fap", axes, sel)
    score = _area(proj.amax(2) - proj.amin(2))
    axes = axes[score.argmin()]
    q = [coords[0] * b[0] + coords[1] * b[1] + coords[2] * b[2] for b in axes]
    low, high = torch.stack([x.amin() for x in q]), torch.stack([x.amax() for x in q])
    if not (score.amin() < _area(hi - lo) and (gpu_rules or _area(high - low) < _area(hi - lo))):
        low, high, axes = lo, hi, torch.eye(3, dtype=axes.dtype, device=axes.device)
    ext = 0.5 * (high - low)
    return torch.cat([0.5 * (low + high) @ axes, axes.flatten(), ext if gpu_rules else ext.clamp(min=0.001)])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fit", "fit_host"):
        box = _box64(_points(case, seed), case.get("gpu_rules", False))
        return box.cpu().numpy() if kind == "fit_host" else box
    # (fit_batch: among thousands of clouds some are needles far from the origin, whose frames are cross products of
    # almost parallel edges: in 32 bits the middle of such a box is off by whole units, so 64 bits say nothing there)
    if kind in ("build", "atrbvh"):
        # the tree hangs on Morton codes rounded in 32 bits; the scene's boxes do not
        m = _mesh(case, seed)
        v = m.verts.double()[m.faces[:, :3].long()]
        lo, hi = v.amin(1), v.amax(1)
        scene = torch.cat([lo.amin(0), hi.amax(0)])
        if kind == "build":
            c = 0.5 * (lo + hi)
            scene = torch.cat([scene, c.amin(0), c.amax(0)])
        out = dict.fromkeys(["nodes", "parents", "counts", "costs", "bounds"])
        out.update(dict.fromkeys(["obbs", "transforms"] if case["obbs"] else []))
        out.update(dict.fromkeys(["collapsed", "primitives"] if case["collapse"] else []))
        out["bounds"] = scene
        return out
    return None
