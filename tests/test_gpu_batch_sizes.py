"""Nearest queries at batch sizes around the walk's own edges: single lanes, a
share per warp below and above the refill threshold, one query more than the
grid's lanes; and answers whose certificate needs the other hits (equal and
nearly equal hits on faces of their own boxes). Bit-exact against the oracle."""
import numpy as np
import pytest

import oracle as O
import spatial_query_b200 as sq
from gpu_util import bits, ctx, pair
from spatial_query_b200 import scenes

pytestmark = pytest.mark.gpu


def leaves(kind, dim, n, seed):
    r = scenes.Rng(seed)
    if kind == "boxes":
        return scenes.boxes_scene(seed=seed, n_boxes=n, n_rays=1, dim=dim)["prims"]
    if kind == "tris":
        return scenes.terrain_scene(seed=seed, nx=64, ny=n // 128, n_coherent=1, n_incoherent=1)["prims"]
    return np.concatenate([r.range(-100.0, 100.0, (n, dim)), r.range(0.25, 4.0, (n, 1))], axis=1)


def rays_for(kind, dim, n, seed):
    r = scenes.Rng(seed)
    if kind == "tris":
        return scenes.terrain_rays(r, 64, 64, -40.0, 40.0, n // 2, n - n // 2)
    return scenes.sphere_rays(r, n, dim)


def same_prefix(ref, h, n):
    assert np.array_equal(ref.leaf[:n], h.leaf), n
    hit = ref.leaf[:n] != O.NO_HIT
    for a, b in ((ref.toi, h.toi), (ref.normal, h.normal), (ref.point, h.point)):
        assert np.array_equal(bits(a[:n][hit]), bits(b[hit])), n


@pytest.mark.parametrize("kind,dim", [("boxes", 2), ("boxes", 3), ("boxes", 4), ("boxes", 6), ("balls", 3),
                                      ("balls_near", 2), ("tris", 3)])
def test_batch_sizes(kind, dim):
    o, g = pair(kind, dim, leaves(kind, dim, 6000, 5))
    rays = rays_for(kind, dim, 200_001, 9)
    ref = o.nearest(rays, 700.0)
    # queries per warp of 148 SMs: 1, 1, 1, 3, 8, 25 and more than its lanes
    for n in (1, 31, 4097, 11_001, 40_000, 131_073, 200_001):
        same_prefix(ref, g.raycast_nearest(rays[:n], 700.0), n)
    r = scenes.Rng(3)
    half = r.range(0.1, 2.0, (11_001, 1)) * np.ones((1, dim), np.float32)
    casts = np.concatenate([rays[:11_001], -half, half], axis=1)
    limits = r.range(50.0, 300.0, 11_001)
    ref = o.shapecast_nearest(casts, limits)
    for n in (31, 11_001):
        same_prefix(ref, g.shapecast_nearest(casts[:n], limits[:n]), n)


@pytest.mark.parametrize("window", [2.0 ** -16, 0.0])
def test_hits_before_their_own_boxes(window):
    """Rays along an axis through the centres of balls that nearly coincide:
    hits lie before their own boxes' entries by rounding, next to hits equal
    to them or a few units in the last place away, and limits cut between."""
    r = scenes.Rng(17)
    n = 4096
    c = r.range(-50.0, 50.0, (n // 8, 3)).repeat(8, axis=0)
    c[:, 0] += np.tile(np.arange(8, dtype=np.float32) % 4, n // 8) * np.float32(2e-6)
    prims = np.concatenate([c, r.range(0.5, 2.0, (n // 8, 1)).repeat(8, axis=0)], axis=1).astype(np.float32)
    o, g = pair("balls", 3, prims)
    origin = c.copy()
    origin[:, 0] = r.range(-190.0, -100.0, n)
    rays = np.concatenate([origin, np.tile(np.array([[1, 0, 0]], np.float32), (n, 1))], axis=1)
    rays[1::2, 3:] = scenes.normalize_rows(np.concatenate([np.ones((n // 2, 1)), r.range(-1e-4, 1e-4, (n // 2, 2))],
                                                          axis=1).astype(np.float32))
    try:
        ctx().set_replay_window(window)
        ref = o.nearest(rays, 400.0)
        assert (ref.leaf != O.NO_HIT).sum() > n // 2
        same_prefix(ref, g.raycast_nearest(rays, 400.0), n)
        limits = ref.toi + np.tile(np.array([0.0, 1e-5, -1e-5, 3e-5], np.float32), n // 4)
        same_prefix(o.nearest(rays, limits), g.raycast_nearest(rays, limits), n)
    finally:
        ctx().set_replay_window(2.0 ** -16)


def scene64(kind, dim, prims):
    geom = sq.Geometry(kind, dim, prims)
    return O.Scene(kind, dim, prims, prec=64), sq.DeviceBvh64(ctx(), sq.HostBvh.build_f64(dim, geom.world_aabbs_f64()),
                                                             geom)


def same64(ref, h, n):
    assert np.array_equal(ref.leaf[:n], h.leaf), n
    hit = ref.leaf[:n] != O.NO_HIT
    assert np.array_equal(ref.toi[:n][hit].view(np.uint64), h.toi[hit].view(np.uint64)), n


@pytest.mark.parametrize("kind,dim", [("boxes", 2), ("boxes", 6), ("balls", 3), ("tris", 3)])
def test_batch_sizes_f64(kind, dim):
    o, g = scene64(kind, dim, leaves(kind, dim, 3000, 5))
    rays = rays_for(kind, dim, 100_001, 9).astype(np.float64)
    ref = o.nearest(rays, 700.0)
    for n in (1, 33, 5000, 100_001):  # thinly dealt, a share per warp, dynamic refill
        same64(ref, g.raycast_nearest(rays[:n], 700.0), n)
    half = np.full((5000, dim), 0.75)
    casts = np.concatenate([rays[:5000], -half, half], axis=1)
    same64(o.shapecast_nearest(casts, 300.0), g.shapecast_nearest(casts, 300.0), 5000)


def test_f64_call_captured_on_a_fresh_context():
    """A first f64 call inside a capture (no replay list yet) is answered."""
    import torch
    fresh = sq.Context(0)
    prims = leaves("balls", 3, 3000, 5)
    geom = sq.Geometry("balls", 3, prims)
    g = sq.DeviceBvh64(fresh, sq.HostBvh.build_f64(3, geom.world_aabbs_f64()), geom)
    rays = rays_for("balls", 3, 3001, 4).astype(np.float64)
    d = torch.from_numpy(rays).cuda()
    leaf, toi = torch.full((3001,), 7, dtype=torch.int32, device="cuda"), torch.zeros(3001, dtype=torch.float64,
                                                                                       device="cuda")
    torch.cuda.synchronize()
    fresh.graph_begin()
    fresh.check(sq.lib().sq_raycast_nearest_f64_d(fresh.h, g.h, d.data_ptr(), 3001, 700.0, None, None, leaf.data_ptr(),
                                                  toi.data_ptr(), None, None), "nearest")
    graph = fresh.graph_end()
    graph.launch()
    fresh.synchronize()
    ref = O.Scene("balls", 3, prims, prec=64).nearest(rays, 700.0)
    same64(ref, sq.Hits(leaf.cpu().numpy().view(np.uint32), toi.cpu().numpy()), 3001)
