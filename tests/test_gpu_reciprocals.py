"""The third-order FP64 reciprocal and reciprocal square root (parrelray_b200/csrc/prr_device.cuh: h3_rcp, h3_rsqrt) by
themselves, over the arguments the kernels feed them.

The correction leaves under 2^-56; the last multiply-add rounds by 2^-53, and 1/sqrt's residual carries half of one more
rounding: under 2^-52 in all (a NaN fails the comparison)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_third_order_forms_against_correct_rounding(gpu):
    rng = np.random.default_rng(15)
    x = np.concatenate([10.0 ** rng.uniform(-12, 12, 400_000), 2.0 ** np.arange(-40.0, 41.0), np.nextafter(2.0 ** np.arange(-40.0, 41.0), 0.0)])
    got = gpu.check_recip_h3(x)
    xl = x.astype(np.longdouble)
    for k, ref in enumerate((1 / xl, 1 / np.sqrt(xl))):
        assert (np.abs(got[:, k].astype(np.longdouble) / ref - 1) <= 2.0**-52).all()
