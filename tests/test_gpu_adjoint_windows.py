"""The adjoint's stored windows (parrelray_b200/csrc/k_adjoint.cu: 4096 accepted steps per ray, earlier windows
recomputed from checkpoints) and its warp-wide reverse sweep, against the FP64 host gradient with the bars of
test_gpu_adjoint.py: rays of one window, of a window and a few steps, of several windows; ray counts that are not
a multiple of a warp."""
import numpy as np
import pytest

from test_gpu_adjoint import gpu_adjoint
from test_oracle_gradient import NAMES, grad_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,hmax,max_steps", [(5, 3, 0.1, 10000), (1, 1, 0.1, 10000), (7, 5, 0.05, 4000), (7, 5, 0.02, 20000),
                                               (11, 3, 0.1, 1400)])
def test_windowed_adjoint_matches_host_gradient(gpu, oracle, small_textures, W, H, hmax, max_steps):
    d = grad_frame(W=W, H_=H, samples=1, tol=1e-8)
    d.hmax, d.max_steps = hmax, max_steps
    gpu.upload_textures(small_textures)
    w = np.random.default_rng(5).normal(size=(H, W, 3)).astype(np.float32)
    g_gpu, st = gpu_adjoint(gpu, d, w)
    g_host, _ = oracle.grad(d, small_textures, w, 0)
    assert st.n_math_error == 0 and st.accepted > 0
    for k in range(5):
        assert abs(g_gpu[k] - g_host[k]) <= 1e-5 * np.abs(g_host).max() + 1e-4 * abs(g_host[k]), (NAMES[k], g_gpu, g_host)
