"""Tile binning at the edges of its chunks and windows (needs a GPU).

A frame's lists must hold, per tile, every Gaussian whose rectangle covers the tile in
(depth, index) order. They are recomputed here from the frame's own projected centres,
extents and depths with the reference's float32 rectangle arithmetic
(core/cpu/msplat_cpu.cpp:505-567) and compared exactly.
"""
import numpy as np
import pytest
import torch

from msplat_street_b200 import scenes
from msplat_street_b200.backend import AdamState, BatchItem, Context, GaussianParams
from msplat_street_b200.camera import look_at, prepare_cam
from parity_util import BACKGROUND, C1_LRS

pytestmark = pytest.mark.gpu


def _expected(ctx, cam):
    """(tile_start, tile_end, ids) from the frame's projections."""
    sp = ctx.frame("splats").cpu().numpy().reshape(-1, 12)
    ext = ctx.frame("aabb").cpu().numpy().reshape(-1, 2)
    vis = np.flatnonzero(ctx.frame("radii").cpu().numpy() > 0)
    vis = vis[np.argsort(sp[vis, 9], kind="stable")]
    f = np.float32
    c, r = sp[vis, :2] / f(16), ext[vis] / f(16)
    lim = np.array([cam.tiles_x, cam.tiles_y])
    lo = np.clip(np.trunc(c - r).astype(np.int64), 0, lim)
    hi = np.clip(np.trunc(c + r + f(1)).astype(np.int64), 0, lim)
    w, n = (hi - lo)[:, 0], (hi - lo).prod(1)
    src = np.repeat(np.arange(len(vis)), n)
    k = np.arange(len(src)) - np.repeat(np.cumsum(n) - n, n)
    tile = (lo[src, 1] + k // w[src]) * cam.tiles_x + lo[src, 0] + k % w[src]
    order = np.argsort(tile, kind="stable")
    ends = np.cumsum(np.bincount(tile, minlength=cam.tiles_x * cam.tiles_y))
    return np.concatenate([[0], ends[:-1]]), ends, vis[src[order]]


def _check(ctx, cam):
    start, end, ids = _expected(ctx, cam)
    assert np.array_equal(ctx.frame("tile_start").cpu().numpy(), start)
    assert np.array_equal(ctx.frame("tile_end").cpu().numpy(), end)
    assert np.array_equal(ctx.frame("isect_gid").cpu().numpy(), ids)
    return len(ids)


# (Gaussians, width, height, log-scale mean): one, and around the 256-Gaussian chunks;
# frames of one tile, of one row, of more tiles than a window holds (8192: 132 x 69),
# and wider than a window (8194 tiles in a row); splats of a few tiles and of hundreds
SIZES = [(1, 16, 16, -3.0), (255, 300, 40, -3.0), (256, 64, 300, -2.0), (257, 16, 16, -1.0),
         (40_000, 2100, 1100, -4.0), (700, 131_100, 20, -2.0), (3000, 640, 480, -1.0)]


@pytest.mark.parametrize("n,w,h,scale", SIZES)
def test_lists_match_the_rectangles(n, w, h, scale):
    p = GaussianParams.from_numpy(scenes.random_gaussians(n, n, log_scale_mean=scale))
    cam = prepare_cam(look_at((0.2, 0.1, 2.6), (0, 0, 0)), w, h, 0.9 * min(w, 2000), 0.9 * min(w, 2000), w / 2.0, h / 2.0)
    ctx = Context()
    for _ in range(2):  # the first frame grows the buffers, the second fits them
        img = ctx.render(p, cam, BACKGROUND)
        assert _check(ctx, cam) > 0
    batch = ctx.render_batch([BatchItem(p, cam, BACKGROUND), BatchItem(p, scenes.small_camera(70, 50), BACKGROUND)])
    assert torch.equal(batch[0], img)


@pytest.mark.parametrize("n", [33, 2049, 16_384, 16_385, 20_480, 20_481, 32_800, 65_536, 65_537, 300_000])
def test_equal_depths_keep_index_order(n):
    """Five distinct depths, so that nearly every neighbour in the depth order is a tie,
    at the sizes where the depth sort changes form (one cluster of blocks, with two and
    four keys a thread, up to 20,480; several launches a digit beyond)."""
    rng = np.random.default_rng(n)
    g = scenes.random_gaussians(n, n, log_scale_mean=-4.5)
    g.means[:, 2] = rng.integers(0, 5, n).astype(np.float32) * 0.25
    g.opacities[rng.random(n) < 0.1] = -20.0
    g.means[rng.random(n) < 0.2, 2] = 9.0  # behind the camera
    cam = prepare_cam(look_at((0.0, 0.0, 3.0), (0.0, 0.0, 0.0)), 400, 240, 300.0, 300.0, 200.0, 120.0)
    ctx = Context()
    ctx.render(GaussianParams.from_numpy(g), cam, BACKGROUND)
    assert _check(ctx, cam) > 0


def test_no_visible_gaussian():
    """Every Gaussian behind the camera: empty lists, the background everywhere."""
    p = GaussianParams.from_numpy(scenes.random_gaussians(1000, 1))
    cam = prepare_cam(look_at((0.0, 0.0, 3.0), (0.0, 0.0, 9.0)), 100, 60, 90.0, 90.0, 50.0, 30.0)
    ctx = Context()
    img = ctx.render(p, cam, BACKGROUND)
    assert ctx.num_isects() == 0 and int(ctx.frame("tile_end").max()) == 0
    assert torch.equal(img, torch.from_numpy(BACKGROUND).cuda().expand_as(img))


@pytest.mark.parametrize("nv", [1, 3, 9])
def test_batched_step_lists(nv):
    """A batched step of several views against the sum of single-view gradients: the
    view-major depth order (one pass more from two views on) and the shared lists."""
    g = scenes.random_gaussians(700, 3, log_scale_mean=-2.5)
    cams = [prepare_cam(look_at((0.3 * v - 1, 0.2, 2.6), (0, 0, 0)), 60 + 17 * v, 90 - 7 * v, 70.0, 70.0,
                        30.0 + 8 * v, 45.0 - 3 * v) for v in range(nv)]
    gts = [torch.rand((c.height, c.width, 3), device="cuda") for c in cams]
    ctx, p = Context(), GaussianParams.from_numpy(g)
    grads = [torch.zeros_like(t) for t in p.tensors()]
    losses = ctx.train_batch(p, None, list(zip(cams, gts)), BACKGROUND, grads=grads)
    total = [torch.zeros_like(t) for t in grads]
    for v, (c, gt) in enumerate(zip(cams, gts)):
        one = [torch.zeros_like(t) for t in p.tensors()]
        assert ctx.train_batch(p, None, [(c, gt)], BACKGROUND, grads=one)[0] == losses[v]
        total = [a + b for a, b in zip(total, one)]
    for a, b in zip(grads, total):
        assert torch.equal(a, b)  # added view by view in both


@pytest.mark.parametrize("n,w,h", [(3000, 592, 256), (3000, 9488, 16), (1, 1000, 500), (4000, 2048, 1024),
                                   (4000, 2064, 1024)])
def test_ordered_tiles_change_no_step(n, w, h):
    """Frames around the tile counts whose blocks take the tiles by list length (593 to
    8192; 592 and 8256 go by index; the one of a single Gaussian is mostly empty): two
    steps equal the batched step's, whose tiles go by index, bit for bit."""
    g = scenes.random_gaussians(n, 3 * n + w, log_scale_mean=-2.5)
    cam = prepare_cam(look_at((0.2, 0.1, 2.6), (0, 0, 0)), w, h, 0.8 * h + 64, 0.8 * h + 64, w / 3.0, h / 2.0)
    gt = torch.rand((h, w, 3), generator=torch.Generator().manual_seed(n)).cuda()
    sides = []
    for batch in (False, True):
        p = GaussianParams.from_numpy(g)
        adam = AdamState.zeros_like(p, C1_LRS)
        stats = tuple(torch.zeros(n, device="cuda") for _ in range(3))
        ctx = Context()
        for _ in range(2):
            if batch:
                loss = float(ctx.train_batch(p, adam, [(cam, gt)], BACKGROUND, stats)[0])
            else:
                loss = ctx.train_step(p, adam, cam, BACKGROUND, gt, stats, sync_loss=True)
        sides.append((loss, p.tensors() + adam.exp_avg + adam.exp_avg_sq + list(stats)))
    assert sides[0][0] == sides[1][0]
    for x, y in zip(sides[0][1], sides[1][1]):
        assert torch.equal(x, y)
