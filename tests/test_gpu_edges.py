"""Edge cases of the plain path against the CPU oracle (needs a GPU): an empty scene,
every Gaussian behind the camera, one-pixel and one-row images, a Gaussian covering
the whole image, saturated opacities (alpha capped at 0.999, early termination), and
SH degree 0. Bars as the plain parity tests: integer data bit-exact, images max-abs
<= 1e-5, gradients relative L2 <= 1e-4."""
import numpy as np
import pytest
import torch

from msplat_street_b200 import autograd, scenes
from msplat_street_b200.backend import AdamState, Context, GaussianParams
from msplat_street_b200.camera import look_at, prepare_cam
from oracle_lib import Oracle, new_adam_state
from parity_util import BACKGROUND, C1_LRS, GRAD_RTOL_L2, IMAGE_ATOL, max_abs, rel_l2

pytestmark = pytest.mark.gpu

GRAD_KEYS = ("v_xy", "v_conic", "v_rgb", "v_opacity", "v_mean3d", "v_scale", "v_quat")


@pytest.fixture(scope="module")
def oracle():
    return Oracle("restatement")


def _empty(deg=3):
    z = np.zeros((0, 3), np.float32)
    return scenes.Gaussians(z, z, np.zeros((0, 4), np.float32), z, np.zeros((0, (deg + 1) ** 2 - 1, 3), np.float32),
                            np.zeros((0, 1), np.float32))


def _saturated(n=800, seed=3):
    g = scenes.random_gaussians(n, seed, log_scale_mean=-2.5)
    g.opacities[:] = 8.0  # sigmoid ~ 0.9997: alpha capped at 0.999, pixels terminate early
    return g


def _huge(seed=4):
    g = scenes.random_gaussians(50, seed, log_scale_mean=-4.0)
    g.means[0] = 0.0
    g.scales[0] = np.log(3.0)  # wider than the whole view
    g.opacities[0] = -1.0
    return g


def _behind(n=500, seed=5):
    g = scenes.random_gaussians(n, seed)
    g.means[:, 2] += 10.0  # the camera sits at z = 3 looking down -z: everything behind it
    return g


CASES = {
    "empty": (_empty, lambda: scenes.small_camera(64, 48, 80.0)),
    "behind_camera": (_behind, lambda: scenes.small_camera(64, 48, 80.0)),
    "one_pixel": (lambda: scenes.random_gaussians(300, 6, log_scale_mean=-2.0), lambda: scenes.small_camera(1, 1, 2.0)),
    "one_row": (lambda: scenes.random_gaussians(400, 7, log_scale_mean=-2.5), lambda: scenes.small_camera(37, 1, 30.0)),
    "huge": (_huge, lambda: prepare_cam(look_at((0.2, 0.1, 2.0), (0, 0, 0)), 80, 60, 70.0, 70.0, 40.0, 30.0)),
    "saturated": (_saturated, lambda: scenes.small_camera(96, 64, 110.0)),
    "sh_degree_0": (lambda: scenes.random_gaussians(1500, 8, sh_degree=0), lambda: scenes.small_camera(80, 80, 100.0)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_render_edge(oracle, name):
    make_g, make_cam = CASES[name]
    g, cam = make_g(), make_cam()
    img_o = oracle.render(g, cam, BACKGROUND)
    ctx = Context()
    img = ctx.render(GaussianParams.from_numpy(g), cam, BACKGROUND).cpu().numpy()
    assert max_abs(img, img_o) <= IMAGE_ATOL
    for key in ("tile_start", "tile_end", "final_idx"):
        assert np.array_equal(ctx.frame(key).cpu().numpy(), oracle.frame(key)), key
    if g.n:
        assert np.array_equal(ctx.frame("radii").cpu().numpy(), oracle.frame("radii"))
    if name in ("empty", "behind_camera"):
        assert np.array_equal(img, np.broadcast_to(np.clip(BACKGROUND, 0, 1), img.shape))
        assert ctx.num_isects() == 0


@pytest.mark.parametrize("name", sorted(CASES))
def test_train_step_edge(oracle, name):
    make_g, make_cam = CASES[name]
    g, cam = make_g(), make_cam()
    gt = np.random.default_rng(1).random((cam.height, cam.width, 3)).astype(np.float32)
    go = g.copy()
    ad = new_adam_state(go, C1_LRS, 1)
    ad["m1"] = [np.full_like(a, 0.01) for a in g.arrays()]  # nonzero moments: every Gaussian's decay shows
    ad["m2"] = [np.full_like(a, 0.02) for a in g.arrays()]
    st = {k: np.zeros(g.n, np.float32) for k in ("vis", "gn", "ms")}
    loss_o = oracle.train_step(go, cam, BACKGROUND, gt, ad, st)
    ctx = Context(keep_grads=True)
    p = GaussianParams.from_numpy(g)
    adam = AdamState.zeros_like(p, C1_LRS)
    for t in adam.exp_avg:
        t.fill_(0.01)
    for t in adam.exp_avg_sq:
        t.fill_(0.02)
    stats = tuple(torch.zeros(g.n, device="cuda") for _ in range(3))
    loss = ctx.train_step(p, adam, cam, BACKGROUND, torch.from_numpy(gt).cuda(), stats, sync_loss=True)
    assert abs(loss - loss_o) <= 1e-6 * max(1.0, abs(loss_o)), (loss, loss_o)
    if g.n == 0:
        return
    for key in GRAD_KEYS:
        got, ref = ctx.frame(key).cpu().numpy(), oracle.frame(key)
        if not np.any(ref):
            assert not np.any(got), key  # nothing visible: exactly zero
        else:
            assert rel_l2(got, ref) <= GRAD_RTOL_L2, (key, rel_l2(got, ref))
    # the Adam step: updates compared as vectors (each element moves by about its
    # learning rate whatever its gradient), moments and statistics likewise
    for before, gpu, ref, nm in zip(g.arrays(), p.numpy(), go.arrays(),
                                    ("means", "scales", "quats", "dc", "rest", "opacities")):
        d_gpu, d_ref = gpu.reshape(ref.shape) - before, ref - before
        if np.any(d_ref):
            assert rel_l2(d_gpu, d_ref) <= 1e-3, nm
        else:
            assert not np.any(d_gpu), nm
    for gpu, ref in zip(adam.exp_avg + adam.exp_avg_sq, ad["m1"] + ad["m2"]):
        assert rel_l2(gpu.cpu().numpy().reshape(ref.shape), ref) <= GRAD_RTOL_L2
    assert np.array_equal(stats[0].cpu().numpy(), st["vis"])
    assert rel_l2(stats[1].cpu().numpy(), st["gn"]) <= GRAD_RTOL_L2
    assert np.array_equal(stats[2].cpu().numpy(), st["ms"])


@pytest.mark.parametrize("n,scale,degree", [(1, -1.0, 3), (127, -2.0, 1), (129, -1.0, 2), (300, 0.0, 3)])
def test_slot_sums_of_every_size(n, scale, degree):
    """Screen-space gradients (the sums of the intersection slots) of scenes whose Gaussians
    cover from one tile to the whole 40 x 30 tile frame (sums of one lane, of four, of a
    warp and of the block) and whose counts lie around the backward kernel's 128-Gaussian
    blocks, against the oracle within the gradient tolerance; the batched step's parameters
    and moments are the same bits. (The world-space gradients of such needles are no
    measure of a sum: the covariance VJP turns the projection's one-ulp differences into
    1e-3.)"""
    rng = np.random.default_rng(n)
    g = scenes.random_gaussians(n, n, sh_degree=degree, log_scale_mean=scale, log_scale_std=1.5)
    cam = scenes.small_camera(640, 480, 500.0)
    gt = rng.random((480, 640, 3)).astype(np.float32)
    oracle = Oracle("restatement")
    go = g.copy()
    oracle.train_step(go, cam, BACKGROUND, gt, new_adam_state(go, C1_LRS, 1),
                      {k: np.zeros(n, np.float32) for k in ("vis", "gn", "ms")}, degrees_to_use=degree)
    ctx, gt_t = Context(keep_grads=True), torch.from_numpy(gt).cuda()
    p, q = GaussianParams.from_numpy(g), GaussianParams.from_numpy(g)
    ap, aq = AdamState.zeros_like(p, C1_LRS), AdamState.zeros_like(q, C1_LRS)
    ctx.train_step(p, ap, cam, BACKGROUND, gt_t, None, degrees_to_use=degree)
    for key in ("v_xy", "v_conic", "v_rgb", "v_opacity"):
        got, ref = ctx.frame(key).cpu().numpy(), oracle.frame(key)
        assert rel_l2(got, ref) <= GRAD_RTOL_L2, (key, rel_l2(got, ref))
    ctx.train_batch(q, aq, [(cam, gt_t)], BACKGROUND, degrees_to_use=degree)
    for a, b in zip(p.tensors() + ap.exp_avg + ap.exp_avg_sq, q.tensors() + aq.exp_avg + aq.exp_avg_sq):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n,degree,unseen", [(1, 3, 0.0), (127, 0, 0.5), (128, 3, 0.0), (129, 2, 0.5), (1000, 3, 0.9),
                                             (1000, 1, 0.0)])
def test_gradients_with_and_without_the_update(n, degree, unseen):
    """The backward that writes gradients and the one that also updates are two kernels:
    the same gradients bit for bit, in blocks all visible, mixed and ragged."""
    g = scenes.random_gaussians(n, n, sh_degree=degree, log_scale_mean=-2.5)
    g.means[np.random.default_rng(n).random(n) < unseen, 2] += 10.0  # behind the camera
    cam = scenes.small_camera(160, 120, 130.0)
    gt = torch.rand((120, 160, 3), device="cuda")
    frames, moments = [], None
    for update in (True, False):
        ctx, p = Context(keep_grads=True), GaussianParams.from_numpy(g)
        adam = AdamState.zeros_like(p, C1_LRS)
        stats = [torch.zeros(n, device="cuda") for _ in range(3)]
        ctx.train_step(p, adam, cam, BACKGROUND, gt, stats, num_adam_groups=6 if update else 0)
        frames.append([ctx.frame(k).clone() for k in GRAD_KEYS] + stats)
        moments = adam.exp_avg if update else moments
    for a, b in zip(*frames):
        assert torch.equal(a, b)
    seen = frames[0][-3] > 0
    assert bool(seen.any()) and (unseen == 0 or not bool(seen.all()))
    p = GaussianParams(*[torch.from_numpy(a).cuda().requires_grad_(True) for a in g.arrays()])
    autograd.ssim_l1_loss(autograd.render(p, cam, BACKGROUND), gt).backward()
    for t, m in zip(p.tensors(), moments):  # the first moments of one step from zero
        if t.numel():
            assert torch.allclose(t.grad.reshape(m.shape) * np.float32(1.0 - np.float32(0.9)), m, rtol=1e-6, atol=0)


def _half_up(x):
    """float64 -> float32 (nearest) -> half (toward +infinity), as the record is packed."""
    f = x.astype(np.float32)
    with np.errstate(over="ignore"):
        h = f.astype(np.float16)
    return np.where(h.astype(np.float32) < f, np.nextafter(h, np.float16(np.inf)), h)


def test_skip_extents_in_64_bits():
    """The four extents of every visible Gaussian's record are the 64-bit ones of its conic
    and opacity (a Gaussian that can reach no pixel has an empty box)."""
    g = scenes.random_gaussians(200_000, 9, log_scale_mean=-4.0, log_scale_std=1.0)
    g.opacities[:] = np.random.default_rng(9).normal(-4.0, 2.0, g.opacities.shape)
    ctx = Context()
    ctx.render(GaussianParams.from_numpy(g), scenes.small_camera(512, 384, 400.0), BACKGROUND)
    rec = ctx.frame("splats").cpu().numpy().reshape(g.n, 12)[ctx.frame("radii").cpu().numpy() > 0]
    a, b, c, op = (rec[:, k].astype(np.float64) for k in (2, 3, 4, 5))
    got = np.ascontiguousarray(rec[:, 10:12]).view(np.float16)
    lg, det = np.log(255.0 * op), a * c - b * b
    reach, diag = np.minimum(5.55, lg + 1e-4), np.minimum(5.55, lg) + 1e-2
    assert (det > 0).all() and (reach <= 0).any() and (diag <= 0).any()

    def extent(level, num, none):
        return np.where(level > 0, np.sqrt(np.maximum(2.0 * level * num / det, 0.0)) * 1.001 + 0.5, none)

    want = [extent(reach, c, -np.inf), extent(reach, a, -np.inf), extent(diag, np.maximum(a + c - 2 * b, 0), np.inf),
            extent(diag, np.maximum(a + c + 2 * b, 0), np.inf)]
    assert len(rec) > 100_000
    for k, w in enumerate(want):
        assert np.array_equal(got[:, k], _half_up(w)), k
