"""The launch shape of a context that nobody tuned (parrelray_b200/csrc/render.cu:launch_shape): the CTA size of the
kernel that renders, on both sides of the 2048 pixels per SM; a shape that was set is used as it is; images do not
depend on it."""
import numpy as np
import pytest

from parrelray_b200 import Context, Graph, LaunchConfig, abi
from test_gpu_work_items import frame

pytestmark = pytest.mark.gpu
F32, F64, SPLIT = abi.PREC_FP32, abi.PREC_FP64, abi.PREC_SPLIT


@pytest.mark.parametrize("hamiltonian,table,precision,w,h,block", [
    (3, -1, F32, 64, 36, 64), (3, -1, F64, 64, 36, 64), (3, -1, SPLIT, 64, 36, 64), (3, 1, F32, 64, 36, 64),
    (0, -1, F32, 64, 36, 128), (0, -1, F32, 592, 512, 128), (0, -1, F32, 592, 513, 64), (0, -1, SPLIT, 64, 36, 128),
    (0, -1, F64, 64, 36, 128), (0, 1, F64, 592, 513, 128), (0, 1, F32, 64, 36, 64), (1, -1, F64, 64, 36, 128)])
def test_untuned_cta_size(small_textures, hamiltonian, table, precision, w, h, block):
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes for 148 SMs")
    d = frame(w, h, 1, precision=precision)
    d.max_steps = 200
    out = torch.zeros(w * h * 3, dtype=torch.uint8, device="cuda")
    with Context(0) as ctx:
        ctx.upload_textures(small_textures)
        ctx.set_option(abi.OPT_HAMILTONIAN, hamiltonian)
        ctx.set_option(abi.OPT_GEOD_TABLE, table)
        with Graph(ctx, [d], out.data_ptr()) as g:
            assert g.launch_config().block_size == block
        img, _, _ = ctx.render(d)
        ctx.set_schedule(abi.SCHED_PERSISTENT, LaunchConfig(64, 0, 64, 1))
        with Graph(ctx, [d], out.data_ptr()) as g:
            assert g.launch_config().block_size == 64
            g.launch()
            g.stats()
        assert np.array_equal(out.cpu().numpy(), img[0].ravel())
