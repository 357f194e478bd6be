"""The adjoint's stored windows (parrelray_b200/csrc/render.cu:prr_adjoint, k_adjoint.cu) at lengths set by
PRR_OPT_ADJOINT_WINDOW and under scarce device memory, and the fall back from rays to pixels as work items there.

A window decides only which steps are recomputed, from states the same code stored: the gradient is the same up to
the order of its FP64 sums over rays.  At most 2000 of them follow one another (1800 warps' totals and a lane's rays) and
their terms add up to some 250 times the result (60,000 rays of random sign): 2000 x 250 x 2^-53 < 1e-10."""
import numpy as np
import pytest

from parrelray_b200 import Context, abi, scenes
from test_gpu_adjoint import gpu_adjoint
from test_gpu_work_items import frame
from test_oracle_gradient import grad_frame

pytestmark = pytest.mark.gpu


def close(g, ref):
    return np.abs(g - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("precision", [abi.PREC_FP32, abi.PREC_FP64])
@pytest.mark.parametrize("W,H,hmax", [(7, 5, 0.1), (5, 3, 0.02)])
def test_gradient_does_not_depend_on_the_window(small_textures, precision, W, H, hmax):
    """Windows that hold every ray, that miss one by a step or two, and that it crosses many times."""
    d = grad_frame(W=W, H_=H, samples=1, tol=1e-6)
    d.precision, d.hmax, d.max_steps = precision, hmax, 20000
    w = np.random.default_rng(5).normal(size=(H, W, 3)).astype(np.float32)
    with Context(0) as ctx:
        ctx.upload_textures(small_textures)
        n = int(ctx.trace_rays(d)[0][:, 11].max())  # near the longest ray of the adjoint's own forward steps
        ctx.set_option(abi.OPT_ADJOINT_WINDOW, 3 * n)
        ref, st0 = gpu_adjoint(ctx, d, w)
        assert st0.n_math_error == 0 and st0.accepted > 0 and np.abs(ref).max() > 0
        for window in [64, 333, n // 2, n - 1, n, n + 1, n + 2, 0]:
            ctx.set_option(abi.OPT_ADJOINT_WINDOW, window)
            g, st = gpu_adjoint(ctx, d, w)
            assert st.n_math_error == 0 and st.accepted == st0.accepted, window
            assert close(g, ref), (window, g, ref)


def test_window_option_range(gpu):
    for bad in (-1, (1 << 20) + 1):
        with pytest.raises(abi.PrrError):
            gpu.set_option(abi.OPT_ADJOINT_WINDOW, bad)


class Filled:
    """Leaves `spare` bytes of device memory free."""

    def __init__(self, spare):
        import torch

        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.buf = torch.empty(free - spare, dtype=torch.uint8, device="cuda") if free > spare else None

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch

        self.buf = None
        torch.cuda.empty_cache()


@pytest.mark.parametrize("precision,mib", [(abi.PREC_FP32, 3000), (abi.PREC_FP32, 1080), (abi.PREC_FP32, 800), (abi.PREC_FP32, 400),
                                           (abi.PREC_FP64, 1500), (abi.PREC_FP64, 700)])
def test_gradient_with_little_memory(small_textures, precision, mib):
    """From a window of some thousand steps to fewer threads than a wave: max_steps of 10000 asks for many checkpoints.
    A large wave (300 x 200 rays) and the same gradient as with all of the memory."""
    d = grad_frame(W=300, H_=200, samples=1, tol=1e-6)
    d.precision, d.max_steps = precision, 10000
    w = np.random.default_rng(6).normal(size=(200, 300, 3)).astype(np.float32)
    with Context(0) as ctx:
        ctx.upload_textures(small_textures)
        ref, st0 = gpu_adjoint(ctx, d, w)
    with Context(0) as ctx:
        ctx.upload_textures(small_textures)
        ctx.render(d)  # what the forward render needs is allocated
        with Filled(mib << 20):
            for _ in range(2):
                g, st = gpu_adjoint(ctx, d, w)
                assert st.n_math_error == 0 and st.accepted == st0.accepted
                assert close(g, ref), (g, ref)


def test_gradient_leaves_three_quarters_of_the_memory(small_textures):
    import torch

    d = grad_frame(W=300, H_=200, samples=1, tol=1e-6)
    d.max_steps = 10000
    w = np.ones((200, 300, 3), dtype=np.float32)
    with Context(0) as ctx, Filled(12 << 30):
        ctx.upload_textures(small_textures)
        ctx.render(d)
        before = torch.cuda.mem_get_info()[0]
        gpu_adjoint(ctx, d, w)
        after = torch.cuda.mem_get_info()[0]
        assert after >= 0.74 * before, (before, after)
        # and what it keeps for its next gradient is given back to a call of the context that needs it
        with Filled(64 << 20):
            big = frame(5000, 4000, 1)
            big.max_steps = 3
            ctx.render(big)


def test_frames_without_room_for_ray_colours_render_pixel_by_pixel(small_textures):
    """4096x2048 with 16 samples: 1.6 GB of per-ray colours where 1.2 GB are free; five steps a ray."""
    d = frame(4096, 2048, 16)
    d.max_steps, d.nspheres = 5, 0
    d.rout = 17.9  # inside the camera's 18: a ray shows the sky after its first step
    with Context(0) as ctx:
        ctx.upload_textures(small_textures)
        ref, _, st0 = ctx.render(d)
    with Context(0) as ctx, Filled(1200 << 20):
        ctx.upload_textures(small_textures)
        img, _, st = ctx.render(d)
        assert st.kernel_launches < st0.kernel_launches  # no combine pass
        assert st.attempts == st0.attempts and st.n_escaped == st0.n_escaped and st.n_infinite == st0.n_infinite
        assert np.array_equal(img[0], ref[0])
