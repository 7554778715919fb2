"""The query path's workloads, from single calls of a few rays to whole frames.

Each case is a dict of plain values; ``family`` names the call it makes, and
the other entries its sizes and options. ``prepare`` uploads the scene and the
queries a program would hold before the call, ``run`` makes one pass through
the package's public entry points and returns every output, ``exact`` answers
the same queries by brute force in 64 bits with plain torch where that is
affordable.

Scenes are the repository's own (``scenes.py``): axis-aligned boxes and balls
seen from a sphere shell, a height-field of triangles, a D = 6 Gaussian
mixture of boxes, and 4,096 instances of 16 meshes. A program keeps its scene
and sends new queries, so a scene depends on the case alone and the queries
(and the deformations, translations and training batches) on the seed.
"""
from __future__ import annotations

import functools
import math
from types import SimpleNamespace

import numpy as np
import torch

import spatial_query_b200 as sq
from spatial_query_b200 import scenes

MASK = 0x5  # the layer mask of filtered cases: leaves carry one of four layers, half of them pass
HIDDEN, INPUTS = 128, 6


def listed():
    return [
        # A handful of picking or line-of-sight rays against a small scene: the
        # smallest batch a program sends to the device, where launches count.
        dict(name="rays_few", family="nearest", shape="boxes", dim=3, leaves=10_000, queries=256),
        # GpuRaycaster's own form: rays and hits in host arrays, one blocking call.
        dict(name="rays_host", family="nearest", shape="boxes", dim=3, leaves=10_000, queries=65_536, host=True),
        # The headline batch: 1,048,576 rays, half of them coherent, against the
        # 1,048,576-triangle height field, rays and hits resident on the device.
        dict(name="rays_terrain", family="nearest", shape="tris", dim=3, leaves=1_048_576, queries=1_048_576),
        # The same batch seeded by the learned guide (inference, then the walk).
        dict(name="rays_guided", family="guided", leaves=1_048_576, queries=1_048_576),
        # Every hit along a ray (transparency, thickness): sorted lists of 16.
        dict(name="rays_all", family="all", shape="tris", dim=3, leaves=1_048_576, queries=500_000, k=16),
        # A physics step's swept balls with layer filter and a length per cast.
        dict(name="casts_filtered", family="casts", shape="balls", dim=3, leaves=100_000, queries=100_003,
             layers=True, limits=True),
        # Broad phase / range search in a six-dimensional index, as CSR lists.
        dict(name="overlap_6d", family="overlap", shape="boxes", dim=6, leaves=2_097_152, queries=262_144),
        # A frame of the two-level scene: refit of the moved instances, then one
        # mixed launch of rays, casts and regions, replayed as a CUDA graph.
        dict(name="tlas_frame", family="tlas", instances=4096, meshes=16, rays=1_000_000, casts=262_144,
             regions=262_144),
        # A deforming mesh: the tree is refit to new vertices and queried.
        dict(name="refit_rays", family="refit", shape="tris", dim=3, leaves=1_048_576, queries=262_144),
        # A scene rebuilt on the device because its leaves moved too far to refit.
        dict(name="tree_build", family="build", shape="tris", dim=3, leaves=1_048_576),
        # A large-world program in double precision, host arrays in and out.
        dict(name="rays_f64", family="nearest64", shape="boxes", dim=3, leaves=200_000, queries=100_001),
        # One epoch of the guide's training on labelled rays (16 steps of 8,192).
        dict(name="guide_train", family="train", leaves=131_072, batch=8192, steps=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    family = rng.choice(["nearest", "nearest", "nearest", "all", "casts", "overlap", "overlap", "tlas", "refit",
                         "build", "nearest64", "train", "guided"])
    c = dict(family=family)
    if family in ("nearest", "all", "casts", "overlap", "refit", "build", "nearest64"):
        c["shape"] = rng.choice(["boxes", "balls", "tris"])
        c["dim"] = 3 if c["shape"] == "tris" else rng.choice([2, 3, 3, 4, 6] if c["shape"] == "boxes" else [2, 3, 3, 4])
        c["leaves"] = _log(rng, 1_000, 1_000_000)
        if family != "build":
            c["queries"] = _log(rng, 256, 1_000_000 if family == "nearest" else 250_000)
    if family == "nearest":
        c["host"] = rng.random() < 0.3
    if family == "all":
        c["k"] = rng.choice([4, 8, 16])
    if family in ("nearest", "all", "casts"):
        c["layers"] = rng.random() < 0.3
        c["limits"] = rng.random() < 0.3
    # Dense scenes: few enough queries that about 20 million results come back.
    per_query = 0.0
    if family == "overlap":
        per_query = 50.0 if c["shape"] == "tris" or c["dim"] == 6 else c["leaves"] * (7.0 / 200.0) ** c["dim"]
    if family == "all" and c["shape"] != "tris" and c["dim"] != 6:
        per_query = c["leaves"] * (2.25 / 200.0) ** (c["dim"] - 1)
    if per_query > 1.0:
        c["queries"] = max(64, min(c["queries"], int(2e7 / per_query)))
    if family == "tlas":
        c.update(instances=_log(rng, 200, 4096), meshes=rng.choice([1, 4, 16]), rays=_log(rng, 5_000, 500_000),
                 casts=_log(rng, 1_000, 200_000), regions=_log(rng, 1_000, 200_000))
    if family == "train":
        c.update(leaves=_log(rng, 20_000, 200_000), batch=128 * rng.randint(8, 64), steps=rng.randint(2, 16))
    if family == "guided":
        c.update(leaves=_log(rng, 50_000, 1_000_000), queries=_log(rng, 1_000, 1_000_000))
    return c


# ---------------------------------------------------------------------------
# Scenes and queries
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _context():
    """A program has one context per device."""
    return sq.Context(0)


def _grid(leaves):
    """Height-field cells for about this many triangles, twice as wide as deep."""
    ny = max(2, int(round(math.sqrt(leaves / 4))))
    return max(2, leaves // (2 * ny)), ny


@functools.lru_cache(maxsize=2)
def _scene(shape, dim, leaves, layers=False):
    """(geometry, host tree, facts the queries need) of a case's scene."""
    facts = {}
    if shape == "tris":
        nx, ny = _grid(leaves)
        s = scenes.terrain_scene(seed=1, nx=nx, ny=ny, n_coherent=1, n_incoherent=1)
        prims = s["prims"]
        facts = dict(nx=nx, ny=ny, zrange=s["zrange"], max_toi=s["max_toi"])
    elif dim == 6:
        s = scenes.mixture_scene(seed=3, n_boxes=leaves, n_rays=1, n_regions=1)
        prims = s["prims"]
        facts = dict(max_toi=s["max_toi"])
    elif shape == "boxes":
        s = scenes.boxes_scene(seed=0, n_boxes=leaves, n_rays=1, dim=dim)
        prims = s["prims"]
        facts = dict(max_toi=s["max_toi"])
    else:
        r = scenes.Rng(7)
        prims = np.concatenate([r.range(-100.0, 100.0, (leaves, dim)), r.range(0.25, 2.0, (leaves, 1))], axis=1)
        facts = dict(max_toi=1000.0)
    lay = (np.uint64(1) << (scenes.Rng(11).take(len(prims)) & np.uint64(3))) if layers else None
    geom = sq.Geometry(shape, dim, prims, layers=lay)
    return geom, sq.HostBvh.build(geom), facts


def _geometry(case):
    return _scene(case["shape"], case["dim"], case["leaves"], bool(case.get("layers")))


def _rays(case, facts, n, seed):
    r = scenes.Rng(1_000_003 + seed)
    dim = case.get("dim", 3)
    if "nx" in facts:
        return scenes.terrain_rays(r, facts["nx"], facts["ny"], *facts["zrange"], n // 2, n - n // 2)
    if dim == 6:
        return scenes.rays_from(r.range(0.0, 1.0, (n, dim)), scenes.isotropic(r, n, dim))
    return scenes.sphere_rays(r, n, dim)


def _casts(case, facts, n, seed):
    """(origin, unit direction, probe min, probe max) per cast and its length."""
    r = scenes.Rng(2_000_003 + seed)
    dim = case["dim"]
    if "nx" in facts:
        z0, z1 = facts["zrange"]
        lo, hi, size, length = np.array([0.0, 0.0, z0]), np.array([facts["nx"], facts["ny"], z1 + 40.0]), (0.2, 2.0), 60.0
    elif dim == 6:
        lo, hi, size, length = np.zeros(dim), np.ones(dim), (0.001, 0.01), 0.5
    else:
        lo, hi, size, length = np.full(dim, -100.0), np.full(dim, 100.0), (0.5, 2.0), 200.0
    o = (lo + (hi - lo) * r.unit64((n, dim))).astype(np.float32)
    d = scenes.normalize_rows(scenes.isotropic(r, n, dim))
    h = r.range(*size, (n, 1 if case["shape"] == "balls" else dim)) * np.ones((1, dim), np.float32)
    casts = np.ascontiguousarray(np.concatenate([o, d, -h, h], axis=1), dtype=np.float32)
    return casts, r.range(0.05 * length, length, n), length


def _regions(case, facts, n, seed):
    r = scenes.Rng(3_000_017 + seed)
    dim = case["dim"]
    if "nx" in facts:
        z0, z1 = facts["zrange"]
        lo, hi, size = np.array([0.0, 0.0, z0]), np.array([facts["nx"], facts["ny"], z1]), (0.5, 4.0)
    elif dim == 6:
        lo, hi, size = np.zeros(dim), np.ones(dim), (0.01, 0.05)
    else:
        lo, hi, size = np.full(dim, -100.0), np.full(dim, 100.0), (0.5, 4.0)
    c = (lo + (hi - lo) * r.unit64((n, dim))).astype(np.float32)
    h = r.range(*size, (n, dim))
    return np.ascontiguousarray(np.concatenate([c - h, c + h], axis=1), dtype=np.float32)


def _limits(n, max_toi, seed):
    return scenes.Rng(4_000_037 + seed).range(0.05 * max_toi, max_toi, n)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _hit_buffers(n, dim):
    return dict(leaf=torch.empty(n, dtype=torch.int32, device="cuda"), toi=torch.empty(n, device="cuda"),
                normal=torch.empty((n, dim), device="cuda"))


def _queries(case, facts, seed):
    """(queries, the call's limit, limits per query or None)."""
    n = case["queries"]
    if case["family"] == "casts":
        q, lens, length = _casts(case, facts, n, seed)
        return q, length, lens if case.get("limits") else None
    q = _rays(case, facts, n, seed)
    return q, facts["max_toi"], _limits(n, facts["max_toi"], seed) if case.get("limits") else None


def _deformed(prims, seed):
    """The height field's vertices moved by a wave of the seed's own phase."""
    r = scenes.Rng(5_000_011 + seed)
    a, b = 2.0 * math.pi * r.unit64(2)
    v = prims.reshape(-1, 3, 3).copy()
    v[..., 2] += (3.0 * np.sin(v[..., 0] * 0.05 + a) * np.cos(v[..., 1] * 0.05 + b)).astype(np.float32)
    return v.reshape(-1, 9)


def _moved(geom, seed):
    """New leaf parameters of the same count for a refit."""
    if geom.narrow == "tris":
        return _deformed(geom.prims, seed)
    r = scenes.Rng(5_000_011 + seed)
    step = r.range(-1.0, 1.0, (len(geom.prims), geom.dim)) * np.float32(0.002 if geom.dim == 6 else 1.0)
    p = geom.prims.copy()
    p[:, :geom.dim] += step
    if geom.narrow == "boxes":
        p[:, geom.dim:] += step
    return p


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    ctx = _context()
    f = case["family"]
    s = SimpleNamespace(case=case, ctx=ctx)
    if f == "tlas":
        return _prepare_tlas(s, seed)
    if f in ("guided", "train"):
        return _prepare_guide(s, seed)
    geom, tree, facts = _geometry(case)
    s.mask = MASK if case.get("layers") else None
    if f == "build":
        moved = sq.Geometry(geom.narrow, geom.dim, _moved(geom, seed))
        s.aabbs = _dev(moved.world_aabbs())
        return s
    if f == "nearest64":
        s.scene = sq.DeviceBvh64(ctx, _tree64(case), geom)
        s.q = _rays(case, facts, case["queries"], seed).astype(np.float64)
        s.max_toi = facts["max_toi"]
        return s
    s.scene = sq.DeviceBvh(ctx, tree, geom)
    n, dim = case["queries"], case["dim"]
    if f == "overlap":
        s.q = _dev(_regions(case, facts, n, seed))
        s.offsets = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        # The program's result buffer holds twice what a first batch needed.
        first = _dev(_regions(case, facts, n, 0))
        torch.cuda.synchronize()
        total = s.scene.overlap_d(first, n, s.offsets, None, 0)
        s.leaves = torch.zeros(2 * total + 4096, dtype=torch.int32, device="cuda")
        return s
    q, s.max_toi, lim = _queries(case, facts, seed)
    if case.get("host"):
        s.q, s.limits = q, lim
        return s
    s.q, s.limits = _dev(q), None if lim is None else _dev(lim)
    if f == "all":
        k = case["k"]
        s.out = dict(count=torch.zeros(n, dtype=torch.int32, device="cuda"),
                     leaf=torch.full((n, k), -1, dtype=torch.int32, device="cuda"),
                     toi=torch.zeros((n, k), device="cuda"), normal=torch.zeros((n, k, dim), device="cuda"))
    else:
        s.out = _hit_buffers(n, dim)
    if f == "refit":
        s.prims = _dev(_moved(geom, seed))
    return s


@functools.lru_cache(maxsize=2)
def _tree64_of(shape, dim, leaves):
    geom = _scene(shape, dim, leaves)[0]
    return sq.HostBvh.build_f64(dim, geom.world_aabbs_f64())


def _tree64(case):
    return _tree64_of(case["shape"], case["dim"], case["leaves"])


@functools.lru_cache(maxsize=2)
def _instanced(instances, meshes):
    return scenes.instanced_scene(seed=2, n_instances=instances, n_blas=meshes, n_rays=2, n_casts=1, n_regions=1,
                                  n_frames=1)


def _prepare_tlas(s, seed):
    case, ctx = s.case, s.ctx
    i = _instanced(case["instances"], case["meshes"])
    s.blas = sq.BlasSet(ctx, i["meshes"])
    s.tlas = sq.DeviceTlas(ctx, "mesh", 3, i["rot"], i["trans"], i["scale"], blas_id=i["blas_id"], blas=s.blas)
    r = scenes.Rng(6_000_023 + seed)
    s.trans = _dev(i["trans"] + r.normal64(i["trans"].shape).astype(np.float32))
    nr, nc, no, k = case["rays"], case["casts"], case["regions"], 16
    ni, half = case["instances"], case["rays"] // 2
    pick = lambda n: (r.take(n) % np.uint64(ni)).astype(np.int64)
    o = r.range(-2200.0, 2200.0, (nr, 3))
    aim = i["trans"][pick(half)] + r.range(-30.0, 30.0, (half, 3))
    s.rays = _dev(scenes.rays_from(o, np.concatenate([aim - o[:half], scenes.isotropic(r, nr - half, 3)])))
    co = i["trans"][pick(nc)] + r.range(-300.0, 300.0, (nc, 3))
    ch = r.range(0.5, 5.0, (nc, 3))
    s.casts = _dev(np.concatenate([co, scenes.normalize_rows(scenes.isotropic(r, nc, 3)), -ch, ch], axis=1))
    s.lens = _dev(r.range(0.0, 200.0, nc))
    rc, rh = i["trans"][pick(no)] + r.range(-200.0, 200.0, (no, 3)), r.range(1.0, 50.0, (no, 3))
    s.regions = _dev(np.concatenate([rc - rh, rc + rh], axis=1))
    s.ray_out, s.cast_out = _hit_buffers(nr, 3), _hit_buffers(nc, 3)
    s.count = torch.zeros(no, dtype=torch.int32, device="cuda")
    s.leaves = torch.full((no, k), -1, dtype=torch.int32, device="cuda")

    def frame():
        s.tlas.refit_d(d_trans=s.trans)
        s.tlas.mixed_d(rays=s.rays, n_rays=nr, ray_max_toi=8000.0, ray_out=s.ray_out, casts=s.casts, n_casts=nc,
                       cast_max_toi=0.0, cast_max_toi_per_query=s.lens, cast_out=s.cast_out, regions=s.regions,
                       n_regions=no, region_k=k, region_count=s.count, region_leaves=s.leaves)

    torch.cuda.synchronize()
    frame()  # sizes the context's scratch before the capture
    ctx.synchronize()
    ctx.graph_begin()
    frame()
    s.graph = ctx.graph_end()
    return s


def _prepare_guide(s, seed):
    case, ctx = s.case, s.ctx
    geom, tree, facts = _scene("tris", 3, case["leaves"])
    s.scene = sq.DeviceBvh(ctx, tree, geom)
    s.max_toi = facts["max_toi"]
    if case["family"] == "train":
        n = case["batch"] * case["steps"]
        s.guide = sq.Guide(s.scene, depth=12, batch=case["batch"], seed=seed)
        s.n, s.rays = n, _dev(_rays(case, facts, n, seed))
        s.labels = torch.empty(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        s.guide.label_d(s.rays, n, s.max_toi, s.labels)
        return s
    # a trained guide, as a program loads it with its scene
    n = 1 << 19
    s.guide = sq.Guide(s.scene, depth=12, batch=8192, seed=0)
    rays = _dev(_rays(case, facts, n, 77))
    labels = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    s.guide.label_d(rays, n, s.max_toi, labels)
    s.guide.train_d(rays, labels, n, 2)
    ctx.synchronize()
    s.q = _dev(_rays(case, facts, case["queries"], seed))
    s.out = _hit_buffers(case["queries"], 3)
    return s


def run(s):
    case = s.case
    f, n = case["family"], case.get("queries")
    if f == "nearest" and case.get("host"):
        h = s.scene.raycast_nearest(s.q, s.max_toi if s.limits is None else s.limits, mask=s.mask)
        return dict(leaf=h.leaf.view(np.int32), toi=h.toi, normal=h.normal, point=h.point,
                    sub_object=h.sub_object.view(np.int32))
    if f in ("nearest", "refit"):
        if f == "refit":
            s.scene.refit_d(s.prims)
        s.scene.raycast_nearest_d(s.q, n, s.max_toi, s.out["leaf"], s.out["toi"], s.out["normal"],
                                  d_max_toi=s.limits, mask=s.mask)
        return s.out
    if f == "guided":
        s.guide.raycast_nearest_guided_d(s.q, n, s.max_toi, s.out["leaf"], s.out["toi"], s.out["normal"])
        return s.out
    if f == "all":
        s.scene.raycast_all_d(s.q, n, s.max_toi, case["k"], s.out["count"], s.out["leaf"], s.out["toi"],
                              s.out["normal"], d_max_toi=s.limits, mask=s.mask)
        return s.out
    if f == "casts":
        s.scene.shapecast_nearest_d(s.q, n, s.max_toi, s.out["leaf"], s.out["toi"], s.out["normal"],
                                    d_max_toi=s.limits, mask=s.mask)
        return s.out
    if f == "overlap":
        s.scene.overlap_d(s.q, n, s.offsets, s.leaves, s.leaves.numel())
        return dict(offsets=s.offsets, leaves=s.leaves)
    if f == "tlas":
        s.graph.launch()
        return dict(rays=s.ray_out, casts=s.cast_out, count=s.count, leaves=s.leaves)
    if f == "build":
        return list(sq.tree_build_d(s.ctx, case["dim"], s.aabbs, s.aabbs.shape[0]))
    if f == "nearest64":
        h = s.scene.raycast_nearest(s.q, s.max_toi)
        return dict(leaf=h.leaf.view(np.int32), toi=h.toi, normal=h.normal)
    losses = s.guide.train_d(s.rays, s.labels, s.n, 1)
    return dict(losses=losses, params=s.guide.get_params())


# ---------------------------------------------------------------------------
# work / tolerance
# ---------------------------------------------------------------------------

def _stride(shape, dim):
    return 2 * dim if shape == "boxes" else (9 if shape == "tris" else dim + 1)


def _scene_bytes(shape, dim, leaves, queries, scalar=4):
    """What the queries cannot do without of the scene: one root-to-leaf path
    of child boxes and one leaf's parameters each, and no more than the whole
    scene once."""
    levels = max(1.0, math.log2(max(leaves, 2) / 4))
    record, leaf = 4 * dim * scalar + 8, (_stride(shape, dim) + 1) * scalar
    return min(leaves / 4 * record + leaves * leaf, queries * (levels * record + leaf))


def _walk_flops(dim, leaves, queries):
    return queries * (max(1.0, math.log2(max(leaves, 2) / 4)) * 2 * 6 * dim + 50)


def _network_flops(n_out):
    return 2.0 * (INPUTS * HIDDEN + 2 * HIDDEN * HIDDEN + HIDDEN * n_out)


def work(case):
    f = case["family"]
    if f == "tlas":
        nr, nc, no = case["rays"], case["casts"], case["regions"]
        b = nr * 44 + nc * (52 + 20) + no * (24 + 4 + 64) + case["instances"] * (64 + 24)
        b += _scene_bytes("boxes", 3, case["instances"], nr + nc + no)
        b += _scene_bytes("tris", 3, 105_000 * case["meshes"], nr // 2)
        return dict(bytes=b, flops=_walk_flops(3, case["instances"], nr + nc + no) + _walk_flops(3, 105_000, nr // 2))
    if f == "train":
        n_out = min(4096, 1 << math.ceil(math.log2(case["leaves"] / 4)))
        params = HIDDEN * INPUTS + 3 * HIDDEN + 2 * HIDDEN * HIDDEN + n_out * HIDDEN + n_out
        n = case["batch"] * case["steps"]
        return dict(bytes=n * 28 + case["steps"] * params * 24, flops=3.0 * n * _network_flops(n_out))
    leaves = case["leaves"]
    shape, dim = case.get("shape", "tris"), case.get("dim", 3)
    if f == "build":
        return dict(bytes=leaves * (2 * dim * 4 + 4) + leaves * (2 * dim * 4 + 12), flops=leaves * 4.0 * dim)
    n = case["queries"]
    scalar = 8 if f == "nearest64" else 4
    q = (4 if f == "casts" else 2) * dim * scalar + (4 if case.get("limits") else 0)
    if f == "all":
        o = 4 + case["k"] * (8 + 4 * dim)
    elif f == "overlap":
        o = 8 + 4
    else:
        o = 4 + scalar * (1 + dim) + (dim * 4 + 4 if case.get("host") else 0)
    b = n * (q + o) + _scene_bytes(shape, dim, leaves, n, scalar)
    fl = _walk_flops(dim, leaves, n)
    if f == "refit":
        b += leaves * 4 * (2 * _stride(shape, dim) + dim)
        fl += leaves * 2.0 * dim
    if f == "guided":
        fl += n * _network_flops(4096)
    return dict(bytes=b, flops=fl)


def tolerance(case):
    # Every query's answer is the crate's own, bit for bit; a built tree is the
    # crate's tree. Training sums bf16 products in 32 bits.
    if case["family"] == "train":
        return {"rel": 2e-3, "max": 0.5}
    return "exact"


# ---------------------------------------------------------------------------
# exact: brute force in 64 bits
# ---------------------------------------------------------------------------

MOST_PAIRS = 2.5e10


def _brute_boxes(q, lo, hi, lim, dim):
    o, d = q[:, None, :dim], q[:, None, dim:2 * dim]
    t0, t1 = (lo[None] - o) / d, (hi[None] - o) / d
    near, far = torch.minimum(t0, t1), torch.maximum(t0, t1)
    enter, axis = near.max(dim=2)
    enter = enter.clamp_min(0.0)
    ok = (enter <= far.min(dim=2).values) & (enter <= lim[:, None])
    t, best = torch.where(ok, enter, math.inf).min(dim=1)
    hit = torch.isfinite(t)
    ax = axis.gather(1, best[:, None])
    n = torch.zeros((len(q), dim), dtype=torch.float64, device=q.device)
    n.scatter_(1, ax, -torch.sign(q[:, dim:2 * dim].gather(1, ax)))
    n[~hit | (t == 0)] = 0.0
    return torch.where(hit, t, 0.0), n


def _brute_balls(q, c, r, grow, lim, dim):
    o, d = q[:, :dim], q[:, dim:2 * dim]
    b = (o * d).sum(1)[:, None] - d @ c.T
    oc2 = (o * o).sum(1)[:, None] - 2.0 * (o @ c.T) + (c * c).sum(1)[None]
    rr = r[None] + grow[:, None]
    disc = b * b - (oc2 - rr * rr)
    root = disc.clamp_min(0.0).sqrt()
    t = -b - root
    t = torch.where(t < 0, -b + root, t)
    ok = (disc >= 0) & (t >= 0) & (t <= lim[:, None])
    t, best = torch.where(ok, t, math.inf).min(dim=1)
    hit = torch.isfinite(t)
    n = torch.nn.functional.normalize(o + d * torch.where(hit, t, 0.0)[:, None] - c[best], dim=1)
    return torch.where(hit, t, 0.0), torch.where(hit[:, None], n, 0.0)


def _brute_tris(q, v, lim, dim):
    o, d = q[:, None, :3], q[:, None, 3:6].expand(-1, len(v), -1)
    v0 = v[None, :, :3]
    e1, e2 = (v[:, 3:6] - v[:, :3])[None], (v[:, 6:] - v[:, :3])[None]
    p = torch.linalg.cross(d, e2.expand_as(d))
    det = (e1 * p).sum(2)
    tv = o - v0
    u = (tv * p).sum(2) / det
    w = torch.linalg.cross(tv, e1.expand_as(tv))
    b = (d * w).sum(2) / det
    t = (e2 * w).sum(2) / det
    ok = (det.abs() >= 1e-8) & (u >= 0) & (u <= 1) & (b >= 0) & (u + b <= 1) & (t > 1e-6) & (t <= lim[:, None])
    t, best = torch.where(ok, t, math.inf).min(dim=1)
    hit = torch.isfinite(t)
    n = torch.nn.functional.normalize(torch.linalg.cross(e1[0], e2[0])[best], dim=1)
    return torch.where(hit, t, 0.0), torch.where(hit[:, None], n, 0.0)


def _exact_nearest(case, seed):
    geom, _, facts = _geometry(case)
    n, dim, shape = case["queries"], case["dim"], case["shape"]
    if len(geom.prims) * n > (2e9 if shape == "tris" else MOST_PAIRS):
        return None
    if case["family"] == "casts" and shape == "tris":
        return None  # defined on the triangles' boxes, not on a closed form
    if case["family"] == "casts" and shape == "boxes" and n > 10_000:
        return None
    q, max_toi, lim = _queries(case, facts, seed)
    prims = _moved(geom, seed) if case["family"] == "refit" else geom.prims
    if case.get("layers"):
        prims = prims[(geom.layers & np.uint64(MASK)) != 0]
    p, q = _dev(prims).double(), _dev(q).double()
    lim = torch.full((n,), float(np.float32(max_toi)), dtype=torch.float64, device="cuda") if lim is None else _dev(lim).double()
    toi, normal = [], []
    step = max(1, int(1.5e8 / max(len(p), 1) / (8 if shape == "balls" else 24)))
    for a in range(0, n, step):
        b = q[a:a + step]
        l = lim[a:a + step]
        if shape == "balls":
            grow = b[:, 3 * dim] if case["family"] == "casts" else torch.zeros(len(b), dtype=torch.float64, device="cuda")
            t, nn = _brute_balls(b, p[:, :dim], p[:, dim], grow, l, dim)
        elif shape == "tris":
            t, nn = _brute_tris(b, p, l, dim)
        elif case["family"] == "casts":
            t, nn = zip(*[_brute_boxes(b[i:i + 1], p[:, :dim] - b[i, 3 * dim:], p[:, dim:] - b[i, 2 * dim:3 * dim],
                                       l[i:i + 1], dim) for i in range(len(b))])
            t, nn = torch.cat(t), torch.cat(nn)
        else:
            t, nn = _brute_boxes(b, p[:, :dim], p[:, dim:], l, dim)
        toi.append(t)
        normal.append(nn)
    out = dict(leaf=None, toi=torch.cat(toi), normal=torch.cat(normal))
    if case.get("host"):
        hit = (out["normal"] != 0).any(dim=1) | (out["toi"] > 0)
        out["point"] = torch.where(hit[:, None], q[:, :dim] + q[:, dim:] * out["toi"][:, None], 0.0)
        out["sub_object"] = None
    return out


def _shuffle(n, seed, step):
    """The epoch's order: Fisher-Yates on SplitMix64 (as the guide documents it)."""
    m = (1 << 64) - 1
    st = scenes.Rng(seed ^ ((0x5851F42D4C957F2D * (step + 1)) & m))
    draws = st.take(n)
    perm = list(range(n))
    for k, i in enumerate(range(n, 1, -1)):
        j = int(draws[k]) % i
        perm[i - 1], perm[j] = perm[j], perm[i - 1]
    return torch.tensor(perm, device="cuda")


def _exact_train(case, seed):
    """The same epoch of AdamW in 64 bits, with no rounding of activations."""
    s = _prepare_guide(SimpleNamespace(case=case, ctx=_context()), seed)
    s.ctx.synchronize()
    info = s.guide.info()
    n_out, nb, B = info["n_out"], info["n_buckets"], case["batch"]
    shapes = [(HIDDEN, INPUTS), (HIDDEN,), (HIDDEN, HIDDEN), (HIDDEN,), (HIDDEN, HIDDEN), (HIDDEN,), (n_out, HIDDEN),
              (n_out,)]
    flat = torch.from_numpy(s.guide.get_params()).cuda().double()
    parts = [t.reshape(h).clone().requires_grad_() for t, h in zip(flat.split([math.prod(h) for h in shapes]), shapes)]
    opt = torch.optim.AdamW(parts, lr=1e-3, betas=(0.9, 0.999), eps=1e-8, weight_decay=0.01)
    box = torch.from_numpy(s.scene.tree.bounds[0].astype(np.float64)).cuda()
    rays = s.rays.double()
    x = torch.cat([(rays[:, :3] - box[:3]) / (box[3:] - box[:3]) * 2.0 - 1.0, rays[:, 3:]], dim=1)
    perm = _shuffle(s.n, seed, 0)
    losses = []
    for k in range(case["steps"]):
        pick = perm[k * B:(k + 1) * B]
        h, y = x[pick], s.labels[pick].long()
        for l in range(3):
            h = torch.relu(h @ parts[2 * l].T + parts[2 * l + 1])
        z = (h @ parts[6].T + parts[7])[:, :nb]
        loss = torch.nn.functional.cross_entropy(z, y, ignore_index=-1)
        opt.zero_grad()
        loss.backward()
        opt.step()
        losses.append(float(loss.detach()))
    return dict(losses=torch.tensor([sum(losses) / len(losses)], dtype=torch.float64),
                params=torch.cat([t.detach().reshape(-1) for t in parts]))


def exact(case, seed):
    f = case["family"]
    if f == "train":
        return _exact_train(case, seed)
    if f in ("nearest", "nearest64", "casts", "refit"):
        return _exact_nearest(case, seed)
    return None
