"""Rays against pixels as work items (parrelray_b200/csrc/render.cu:wants_sample_items, k_ham.cu:ham_start): a
context renders frames with several samples ray by ray and combines them in a second pass, prr_render_noalloc pixel
by pixel in registers; images are the same bytes.  Sizes around the tiles of 8 x 4 pixels, sample counts that do and
do not divide a warp, batches that mix both, and the recorded batch."""
import ctypes as C

import numpy as np
import pytest

from parrelray_b200 import Graph, LaunchConfig, abi, scenes
from test_zz_no_alloc import device_textures

pytestmark = pytest.mark.gpu


def frame(w, h, samples, precision=abi.PREC_FP32, ssaa=abi.SSAA_REGULAR, fxaa=False):
    sph = [(*scenes.orbit_point(9.0, 40.0), 1.0, scenes.SPHERE_ID0)]
    d = scenes.make_frame(w, h, r=18.0, incl_deg=75.0, fov_deg=55.0, metric=abi.METRIC_KERR, spin=0.9, samples=samples,
                          fxaa=fxaa, spheres=sph, precision=precision)
    d.ssaa = ssaa if samples > 1 else abi.SSAA_NONE
    d.ssaa_seed = 5
    return d


BATCHES = {
    "one_pixel": [(1, 1, 4)], "row": [(37, 1, 4)], "column": [(1, 29, 9)], "three_rows": [(8, 3, 4)], "tile": [(8, 4, 1)],
    "tile_and_one": [(9, 5, 4)], "odd": [(31, 17, 9)], "many_samples": [(5, 6, 64)], "one_sample": [(33, 18, 1)],
    "mixed": [(17, 9, 4), (16, 8, 1), (7, 5, 9), (12, 13, 1)],
}


@pytest.mark.parametrize("precision", [abi.PREC_FP32, abi.PREC_FP64])
@pytest.mark.parametrize("name", sorted(BATCHES))
def test_rays_and_pixels_as_items_give_the_same_bytes(gpu, small_textures, name, precision):
    import torch

    frames = [frame(*k, precision=precision, fxaa=name == "odd") for k in BATCHES[name]]
    gpu.upload_textures(small_textures)
    saved = gpu.launch_config()
    gpu.set_schedule(abi.SCHED_PERSISTENT, LaunchConfig(64, 0, 64, 1))
    try:
        ref8, reff, st = gpu.render(frames, want_float=True)
        npx = sum(f.width * f.height for f in frames)
        out8 = torch.zeros(npx * 3, dtype=torch.uint8, device="cuda")
        outf = torch.zeros(npx * 3, dtype=torch.float32, device="cuda")
        with Graph(gpu, frames, out8.data_ptr(), outf.data_ptr()) as g:
            g.launch()
            gs = g.stats()
        graph8, graphf = out8.cpu().numpy(), outf.cpu().numpy()
    finally:
        gpu.set_schedule(abi.SCHED_PERSISTENT, saved)
    assert st.rays == sum(f.nrays for f in frames)
    assert st.n_escaped + st.n_captured + st.n_intersection + st.n_infinite + st.n_math_error == st.rays
    assert gs.attempts == st.attempts
    assert np.array_equal(graph8, np.concatenate([a.ravel() for a in ref8]))
    assert np.array_equal(graphf, np.concatenate([a.ravel() for a in reff]))
    keep, ptrs, w, h = device_textures(small_textures)
    out8.fill_(3)
    arr = (abi.FrameDesc * len(frames))(*frames)
    err = C.create_string_buffer(512)
    rc = abi.load().prr_render_noalloc(arr, len(frames), ptrs, w, h, out8.data_ptr(), outf.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream, err, 512)
    assert rc == abi.OK, err.value.decode()
    torch.cuda.synchronize()
    assert np.array_equal(out8.cpu().numpy(), graph8)


def test_split_precision_by_rays_matches_its_samples(gpu, small_textures):
    """SPLIT with several samples: every sample of a split render is the FP32 or the FP64 ray's."""
    gpu.upload_textures(small_textures)
    img = {p: gpu.render(frame(21, 13, 4, precision=p), want_float=True) for p in (abi.PREC_FP32, abi.PREC_FP64, abi.PREC_SPLIT)}
    s = img[abi.PREC_SPLIT][1][0]
    near = np.minimum(np.abs(s - img[abi.PREC_FP32][1][0]).max(-1), np.abs(s - img[abi.PREC_FP64][1][0]).max(-1))
    assert (near <= 1 / 255).mean() >= 0.99
    assert img[abi.PREC_SPLIT][2].n_fp64 > 0
