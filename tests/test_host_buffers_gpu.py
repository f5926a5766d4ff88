"""Host-buffer calls against their device-buffer twins, bit for bit: ray queries
with every mix of pinned and pageable buffers around the staging chunks' sizes,
host images on both sides of the kept image memory, and material updates whose
table entries form runs, gaps and repeats."""
import ctypes as C

import numpy as np
import pytest

import tpt
import tpt_scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 65535, 65537, 131073, 300001])
@pytest.mark.parametrize("in_pinned,out_pinned", [(False, False), (False, True), (True, False), (True, True)])
def test_query_buffers(ctx, n, in_pinned, out_pinned):
    import torch

    s = tpt.Scene(ctx, [tpt_scenes.sphere_soup(3, 64, 12.0)], [tpt_scenes.identity_instance()])
    rays = torch.from_numpy(tpt_scenes.incoherent_rays(n, seed=n, cube=12.0))
    d = rays.cuda()
    want = [torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, device="cuda"),
            torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty((3, n), device="cuda")]
    s.traverse_device(d.data_ptr(), n, 0, *[w.data_ptr() for w in want], torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    if in_pinned:
        rays = rays.pin_memory()
    got = [torch.full_like(w, -7, device="cpu") for w in want]
    if out_pinned:
        got = [g.pin_memory() for g in got]
    for _ in range(2):  # the second call finds the staging buffers in place
        st = tpt.lib().tpt_traverse(ctx.h, s.h, C.c_void_p(rays.data_ptr()), n, 0,
                                    *[C.c_void_p(g.data_ptr()) for g in got])
        assert st == 0
        for g, w in zip(got, want):
            assert torch.equal(g.view(torch.int32), w.cpu().view(torch.int32))


@pytest.mark.parametrize("width,height", [(1, 1), (97, 61), (4096, 2800)])
def test_host_image_equals_device_image(ctx, width, height):
    import torch

    sc = tpt_scenes.cornell_box(2, tpt_scenes.LAMBERT)
    s = tpt.Scene(ctx, sc["meshes"], sc["instances"], materials=sc["materials"])
    job = s.job(sc["camera"], width, height, 1, 1)
    img = torch.empty((height, width, 3), device="cuda")
    s.render_device(job, img.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    host = s.render(sc["camera"], width, height, 1, 1)
    assert np.array_equal(host.view(np.uint32), img.cpu().numpy().view(np.uint32))


@pytest.mark.parametrize("ids", [[0], [0, 1, 2, 3], [3, 4, 5, 1, 5, 6], [6, 5, 4], [2, 2, 3, 3]])
def test_material_runs(ctx, ids):
    sc = tpt_scenes.cornell_box(4)
    s = tpt.Scene(ctx, sc["meshes"], sc["instances"], materials=sc["materials"])
    rng = np.random.default_rng(len(ids))
    new = [dict(sc["materials"][k], base_color=rng.uniform(0.1, 0.9, 3).astype(np.float32)) for k in ids]
    s.set_openpbr(ids, new)
    got = s.render(sc["camera"], 40, 30, 4, 3)
    mats = list(sc["materials"])
    for k, m in zip(ids, new):
        mats[k] = m  # the last entry of a material counts
    fresh = tpt.Scene(ctx, sc["meshes"], sc["instances"], materials=mats)
    assert np.array_equal(got, fresh.render(sc["camera"], 40, 30, 4, 3))
