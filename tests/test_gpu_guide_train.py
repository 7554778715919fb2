"""One training step's gradients against the CPU restatement at the edges of the
products' tiles and the loss kernel: one row tile and many, wide outputs and a
partial last chunk of columns, one chunk only, and batches in which labels are
missing, out of range, all the same or absent altogether."""
import numpy as np
import pytest

import guide_ref as R
import spatial_query_b200 as sq
from spatial_query_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sq.Context(0)
    yield c
    c.close()


SCENES = {"full": (128, 64), "ragged": (20, 18), "one chunk": (8, 6)}


def setup(ctx, scene, batch, seed=3):
    nx, ny = SCENES[scene]
    s = scenes.terrain_scene(seed=5, nx=nx, ny=ny, n_coherent=batch // 2, n_incoherent=batch - batch // 2)
    geom = sq.Geometry("tris", 3, s["prims"])
    dev = sq.DeviceBvh(ctx, sq.HostBvh.build(geom), geom)
    return s, dev, sq.Guide(dev, depth=12, batch=batch, seed=seed)


@pytest.mark.parametrize("scene,batch", [("full", 128), ("full", 640), ("full", 9600), ("ragged", 128),
                                         ("ragged", 1280), ("one chunk", 256), ("one chunk", 20_096)])
@pytest.mark.parametrize("labels", ["hits", "some", "same", "none"])
def test_gradients(ctx, scene, batch, labels):
    if batch * (4096 if scene == "full" else 512) > 2_000_000 and labels in ("same", "none"):
        pytest.skip("covered at the smaller batches")
    s, dev, guide = setup(ctx, scene, batch)
    info = guide.info()
    d_rays = torch.from_numpy(s["rays"].copy()).cuda()
    d_lab = torch.empty(batch, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    guide.label_d(d_rays, batch, s["max_toi"], d_lab)
    ctx.synchronize()
    y = d_lab.cpu().numpy()
    if labels == "some":
        y[::3] = -1
        y[1::7] = info["n_buckets"] + np.arange(len(y[1::7])) % 100
    elif labels == "same":
        y[:] = info["n_buckets"] - 1
    elif labels == "none":
        y[:] = -1
    d_lab.copy_(torch.from_numpy(y))
    torch.cuda.synchronize()
    loss = guide.forward_backward_d(d_rays, d_lab)
    got = R.unpack(guide.get_grads(), info["n_out"])
    root = dev.read_bounds()[0]
    ref_loss, ref = R.loss_and_grads(R.unpack(guide.get_params(), info["n_out"]),
                                     R.features(s["rays"], root[:3], root[3:]), y, info["n_buckets"])
    assert abs(loss - ref_loss) <= 1e-4 * max(1.0, abs(ref_loss))
    for k, want in ref.items():
        # 2e-2: dZ and the activations are rounded to bf16 (2^-9) at points where
        # sums in another order may round the other way, layer upon layer
        err = np.linalg.norm(got[k] - want) / max(np.linalg.norm(want), 1e-30)
        assert err <= 2e-2 or np.linalg.norm(want) == np.linalg.norm(got[k]) == 0.0, (k, err)
    guide.close()
    dev.close()


def test_epoch_equals_its_steps(ctx):
    """train_d (permuted rows, losses read at the end) against train_step_d on
    the same batches in the epoch's own order."""
    batch, steps, seed = 256, 5, 11
    s, dev, a = setup(ctx, "ragged", batch * steps, seed)
    a.close()
    a, b = (sq.Guide(dev, depth=12, batch=batch, seed=seed) for _ in range(2))
    n = batch * steps
    d_rays = torch.from_numpy(s["rays"].copy()).cuda()
    d_lab = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    a.label_d(d_rays, n, s["max_toi"], d_lab)
    ctx.synchronize()
    loss = a.train_d(d_rays, d_lab, n, 1)
    draws = scenes.Rng(seed ^ 0x5851F42D4C957F2D).take(n)  # the epoch's Fisher-Yates shuffle
    perm = list(range(n))
    for k, i in enumerate(range(n, 1, -1)):
        j = int(draws[k]) % i
        perm[i - 1], perm[j] = perm[j], perm[i - 1]
    order = torch.tensor(perm, device="cuda")
    rays, lab = d_rays[order].contiguous(), d_lab[order].contiguous()
    torch.cuda.synchronize()
    each = [b.train_step_d(rays[k * batch:(k + 1) * batch], lab[k * batch:(k + 1) * batch]) for k in range(steps)]
    assert abs(loss[0] - np.mean(each)) <= 1e-5 * abs(loss[0])
    pa, pb = a.get_params(), b.get_params()
    assert np.linalg.norm(pa - pb) <= 1e-4 * np.linalg.norm(pb)  # sums in the L2 differ in their order
    a.close()
    b.close()
    dev.close()
