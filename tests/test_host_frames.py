"""What the C-ABI launches and leaves behind, on a recorded CUDA runtime (fake_cuda.py;
no GPU): a call that fails leaves no frame that a later call would walk, and the options
that results do not show choose the launches they say."""
import ctypes as C

import pytest

import fake_cuda

N, W, H = 1000, 640, 480  # 1200 tiles


def _frame_kernels(cuda):
    return [k for k in cuda.launches() if "raster" in k[0] or "backward" in k[0] or "pair_count" in k[0]]


def _fails_at_every_allocation(cuda):
    """A larger frame after a good one, its allocations failing one after another."""
    k, seen = 0, []
    while True:
        ctx = cuda.context()
        cuda.allocs_left(-1)
        cuda.readback(5000)
        assert cuda.render(ctx, N, W, H) == 0 and cuda.lib.msplat_cuda_num_isects(ctx) == 5000
        assert cuda.render_backward(ctx, N, W, H) == 0
        cuda.readback(50_000_000)
        cuda.allocs_left(k)
        status = cuda.render(ctx, 20 * N, 2 * W, 2 * H)
        cuda.allocs_left(-1)
        if status == 0:
            assert k > 10  # it does allocate
            return seen
        cuda.launches()
        after = [cuda.render_backward(ctx, n, w, h) for n, w, h in ((20 * N, 2 * W, 2 * H), (N, W, H))]
        seen.append((status, after, cuda.pair_counts(ctx), _frame_kernels(cuda)))
        cuda.lib.msplat_cuda_ctx_destroy(ctx)
        k += 1


def test_failed_allocation_leaves_no_frame():
    for k, (status, after, counts, launched) in enumerate(fake_cuda.run(_fails_at_every_allocation)):
        assert status != 0
        assert after == [1, 1], k  # EINVAL: no render of that scene and camera to follow
        assert counts == 0 and launched == [], k


def _batch_fails_at_every_allocation(cuda):
    """The same with a batch of two larger views after the frame."""
    k, seen = 0, []
    while True:
        ctx = cuda.context()
        cuda.allocs_left(-1)
        cuda.readback(5000)
        assert cuda.render(ctx, N, W, H) == 0
        cuda.readback(50_000_000)
        cuda.allocs_left(k)
        status = cuda.render_batch(ctx, 2, 20 * N, 2 * W, 2 * H)
        cuda.allocs_left(-1)
        cuda.launches()
        seen.append((status, cuda.render_backward(ctx, N, W, H), cuda.pair_counts(ctx), _frame_kernels(cuda)))
        cuda.lib.msplat_cuda_ctx_destroy(ctx)
        if status == 0:
            return seen
        k += 1


def test_failed_batch_leaves_no_frame():
    seen = fake_cuda.run(_batch_fails_at_every_allocation)
    assert len(seen) > 10 and seen[-1][0] == 0
    for k, (_, after, counts, launched) in enumerate(seen):
        assert (after, counts, launched) == (1, 0, []), k


def _too_many_entries(cuda, w, h):
    ctx = cuda.context()
    cuda.readback(5000)
    assert cuda.render(ctx, N, W, H) == 0
    cuda.readback(1 << 31)
    status = cuda.render(ctx, N, w, h)
    cuda.launches()
    after = [cuda.render_backward(ctx, N, *s) for s in ((w, h), (W, H))]
    return status, after, cuda.pair_counts(ctx), _frame_kernels(cuda), cuda.lib.msplat_cuda_num_isects(ctx)


@pytest.mark.parametrize("size", [(W, H), (256, 256), (1920, 1088)])
def test_too_many_intersections_leave_no_frame(size):
    status, after, counts, launched, isects = fake_cuda.run(_too_many_entries, *size)
    assert status == 4 and after == [1, 1] and counts == 0 and launched == [] and isects == 0


def _refused(cuda):
    ctx = cuda.context()
    cuda.readback(5000)
    assert cuda.render(ctx, N, W, H) == 0
    view = list(cuda._view(2 * N, W, H, 0))
    view[1] = None  # no means
    status = cuda.lib.msplat_cuda_render(ctx, *view, 64, 64, 64, view[-1], None)
    return status, cuda.render_backward(ctx, N, W, H)


def test_refused_render_keeps_the_frame():
    assert fake_cuda.run(_refused) == (1, 0)


def _forward_blocks(cuda, shape):
    """(blocks, threads) of the single-view forward, and the batched one's threads."""
    ctx = cuda.context()
    if shape is not None:
        assert cuda.lib.msplat_cuda_ctx_set_option(ctx, b"raster_shape", shape) == 0
    cuda.readback(5000)
    assert cuda.render(ctx, N, W, H) == 0 and cuda.render_batch(ctx, 2, N, W, H) == 0
    fwd = [k for k in cuda.launches() if "raster_fwd" in k[0]]
    assert len(fwd) == 2 and "batch" in fwd[1][0]
    return fwd[0][1], fwd[0][3], fwd[1][3]


@pytest.mark.parametrize("shape,blocks", [(None, (2400, 128, 256)), (0, (1200, 256, 256)), (1, (2400, 128, 128)),
                                          (2, (4800, 64, 64))])
def test_raster_shape_chooses_the_blocks(shape, blocks):
    assert fake_cuda.run(_forward_blocks, shape) == blocks


def _densify(cuda, n, rest):
    """Device bytes a densification holds, and its compaction launches."""
    ctx = cuda.context()
    six = (C.c_void_p * 6)(*[64] * 6)
    count = C.c_int()
    assert cuda.lib.msplat_cuda_densify(ctx, n, 4 * n, 2e-4, 0.01, 0.05, 0, 0.1, 0.5, 0.15, 0, 64, 64, 64, 256.0, six,
                                        rest, six, six, 1, C.byref(count)) == 0
    gathers = sum("compact_gather" in k[0] for k in cuda.launches())
    return cuda.lib.msplat_cuda_ctx_device_bytes(ctx), gathers


# per row of 4 n: seven flags, and the widest buffer's floats; a quarter more for growth
@pytest.mark.parametrize("n,rest,widest", [(10_000_000, 0, 4), (10_000_000, 9, 9), (4_000_000, 24, 24),
                                           (4_000_000, 45, 45), (1_000_000, 72, 72)])
def test_densify_scratch_is_the_widest_buffer(n, rest, widest):
    held, _ = fake_cuda.run(_densify, n, rest)
    assert held <= 1.26 * 4 * n * 4 * (7 + widest)


@pytest.mark.parametrize("n,rest,gathers", [(100_000, 0, 1), (100_000, 45, 4), (400_000, 45, 4)])
def test_densify_compacts_narrow_buffers_together(n, rest, gathers):
    held, launched = fake_cuda.run(_densify, n, rest)
    assert launched == gathers
    assert held <= 1.26 * (4 * n * 4 * (7 + rest) + (1 << 28))
