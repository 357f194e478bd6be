"""Launches that do not fill the chip (parrelray_b200/csrc/k_ham.cu:launch_ham): below one full warp per scheduler only
some lanes of a warp take work, below one item per lane only as many CTAs per SM as find work are launched.  Which lane
takes a pixel decides nothing: the image has the same bytes and the same attempts as from one CTA of 32 threads per SM,
where neither rule acts.  Sizes on both sides of each line for 148 SMs (592 and 18,944 items, and a CTA's worth per SM)."""
import numpy as np
import pytest

from parrelray_b200 import LaunchConfig, abi
from test_gpu_work_items import frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP32, abi.PREC_FP64])
@pytest.mark.parametrize("w,h", [(1, 1), (37, 16), (25, 24), (148, 127), (148, 128), (149, 128), (192, 148), (193, 148)])
def test_small_launches_give_the_same_bytes(gpu, small_textures, w, h, precision):
    gpu.upload_textures(small_textures)
    saved = gpu.launch_config()
    out = []
    try:
        for shape in [(32, 1, 64, 1), (64, 0, 64, 1), (96, 0, 1, 1), (256, 0, 64, 1)]:
            gpu.set_schedule(abi.SCHED_PERSISTENT, LaunchConfig(*shape))
            img8, imgf, st = gpu.render(frame(w, h, 1, precision=precision), want_float=True)
            out.append((img8[0], imgf[0], st.attempts, st.accepted, st.rays))
    finally:
        gpu.set_schedule(abi.SCHED_PERSISTENT, saved)
    assert out[0][4] == w * h
    # 96 and 256 threads run another instantiation of the kernel, whose contractions may differ
    assert np.array_equal(out[1][0], out[0][0]) and np.array_equal(out[1][1], out[0][1]) and out[1][2:] == out[0][2:]
    for o in out[2:]:
        assert o[4] == w * h
        assert (np.abs(o[0].astype(int) - out[0][0].astype(int)).max(-1) <= 1).mean() >= 0.99
