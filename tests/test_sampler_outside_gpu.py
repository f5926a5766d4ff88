"""Sampler queries outside the image: a Morton index with bits above the image's
digits has the oracle's values too (a digit's permutation depends on every bit
above it), and depths far beyond a path's."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (7, 5, 3), (128, 128, 16), (640, 480, 64), (1920, 1080, 256),
                                     (4096, 4096, 256), (65536, 2, 1), (4096, 4096, 300)])
def test_queries_outside_the_image(ctx, w, h, spp):
    rng = np.random.default_rng(w + spp)
    n = 1 << 12
    q = rng.integers(0, 1 << 32, (n, 4), dtype=np.uint64).astype(np.uint32)
    q >>= rng.integers(0, 32, (n, 4)).astype(np.uint32)  # any number of bits, in every column
    q[:, 3] >>= 4  # dimensions 2 + 16 depth + .. stay within 32 bits
    q[:64, :2] = [w, h]  # one past the last pixel, and one past the last sample
    q[64:128, 0:3] = [w - 1, h - 1, spp]
    dv, ds = ctx.sampler_values(w, h, spp, q)
    ov, os_ = orc.sampler_values(w, h, spp, q)
    assert np.array_equal(dv.view(np.uint32), ov.view(np.uint32))
    assert np.array_equal(ds, os_)
