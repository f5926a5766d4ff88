"""The sampler's 32-bit index permutation and the 64-bit one beside it: the same
values as the oracle's on both sides of the line (a Morton index of
2 log2(side) + log2(spp) bits, 32 at most for the first), and at the smallest
indices (no digit, a lone last bit, one digit)."""
import numpy as np
import pytest

import oracle as orc
from test_sampler_gpu import queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp", [
    (1, 1, 1), (1, 1, 2), (2, 1, 1), (1, 1, 3), (2, 2, 2), (3, 1, 5),
    (4096, 4096, 256), (8192, 3, 64), (65536, 2, 1),  # 32 bits
    (32768, 5, 2), (4096, 4096, 100),  # 31 bits, an odd number of them
    (4096, 4096, 300), (8192, 3, 128), (65537, 2, 1), (100000, 1, 4096),  # 33, 33, 34 and 46 bits
])
def test_index_permutation_on_both_sides_of_32_bits(ctx, w, h, spp):
    q = queries(w, h, spp, 1 << 12, seed=w + spp)
    dv, ds = ctx.sampler_values(w, h, spp, q)
    ov, os_ = orc.sampler_values(w, h, spp, q)
    assert np.array_equal(dv.view(np.uint32), ov.view(np.uint32))
    assert np.array_equal(ds, os_)
