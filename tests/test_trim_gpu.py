"""`tpt_context_trim` on the device: memory comes back, and the next host-buffer
calls give the same results."""
import numpy as np
import pytest

import tpt
import tpt_scenes

pytestmark = pytest.mark.gpu


def test_calls_after_a_trim():
    import torch

    ctx = tpt.Context(0)
    sc = tpt_scenes.cornell_box(2, tpt_scenes.LAMBERT)
    rays = tpt_scenes.incoherent_rays(1 << 20, seed=4, cube=2.0)

    def calls():
        s = tpt.Scene(ctx, sc["meshes"], sc["instances"], materials=sc["materials"])
        hits = s.closest_hit(rays, want_instance=True)
        return [s.render(sc["camera"], 1024, 1024, 1, 2), hits["t"], hits["prim"], hits["inst"]]

    first = calls()
    free = torch.cuda.mem_get_info()[0]
    ctx.trim()
    # 2^20 rays of 7 planes and 3 outputs, and an image of 2^20 pixels
    assert torch.cuda.mem_get_info()[0] - free >= (1 << 20) * (40 + 12)
    ctx.trim()  # nothing left
    for a, b in zip(first, calls()):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    ctx.close()
