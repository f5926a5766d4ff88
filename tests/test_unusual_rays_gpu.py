"""Ray queries with unusual lanes: zero, negative zero, denormal, huge, infinite and
NaN components.  With finite origins and limits the hits are the oracle's, whatever
the direction holds; with infinite or NaN origins and limits (where minima and
maxima of NaN decide, on which no two machines agree) a query ends without an error,
names triangles of the scene, and gives the same through host and device buffers."""
import numpy as np
import pytest

import tpt
import tpt_scenes
from test_traverse_gpu import build_both

ODD = np.array([0.0, -0.0, 1.0, -1.0, 1e-40, -1e-40, 1e-30, 1e38, -1e38, np.inf, -np.inf, np.nan], np.float32)
SCENES = {"soup": (lambda: {"meshes": [tpt_scenes.sphere_soup(3, 64, 12.0)],
                            "instances": [tpt_scenes.identity_instance()]}, 12.0),
          "cornell": (lambda: tpt_scenes.cornell_box(3), 2.0),
          "grid": (lambda: tpt_scenes.grid_scene(3, 6, 128, 16), 10.0)}


def odd_rays(n, cube, finite):
    """Incoherent rays, about one in seven components replaced by an odd value."""
    rng = np.random.default_rng(n)
    r = tpt_scenes.incoherent_rays(n, seed=n, cube=cube).copy()
    for k in range(7):
        m = rng.random(n) < 0.15
        r[k, m] = rng.choice(ODD[:9] if finite and k in (0, 1, 2) else ODD, m.sum())
    if finite:
        r[6, np.isnan(r[6])] = np.inf
    return r


def same(a, b):
    return (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [tpt.CLOSEST_HIT, tpt.ANY_HIT], ids=["closest", "any"])
@pytest.mark.parametrize("name", list(SCENES))
def test_unusual_directions_match_oracle(ctx, name, mode):
    make, cube = SCENES[name]
    sc = make()
    g, s = build_both(ctx, sc["meshes"], sc["instances"])
    rays = odd_rays(1 << 15, cube, True)
    dev, ref = s.closest_hit(rays, mode, want_instance=True), g.query(rays, mode)
    hit = ref["prim"] >= 0
    assert 0.1 < hit.mean() < 0.9
    assert np.array_equal(dev["prim"], ref["prim"])
    assert np.array_equal(dev["inst"][hit], ref["inst"][hit])
    assert np.all(same(dev["t"], ref["t"]))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [tpt.CLOSEST_HIT, tpt.ANY_HIT], ids=["closest", "any"])
@pytest.mark.parametrize("name", list(SCENES))
def test_unusual_origins_end(ctx, name, mode):
    import torch

    make, cube = SCENES[name]
    sc = make()
    s = tpt.Scene(ctx, sc["meshes"], sc["instances"])
    n = 1 << 15
    rays = odd_rays(n, cube, False)
    host = s.closest_hit(rays, mode, want_instance=True, want_bary=True)
    d = torch.from_numpy(rays).cuda()
    prim, inst = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
    t, bary = torch.empty(n, device="cuda"), torch.empty((3, n), device="cuda")
    s.traverse_device(d.data_ptr(), n, mode, prim.data_ptr(), t.data_ptr(), inst.data_ptr(), bary.data_ptr(),
                      torch.cuda.current_stream().cuda_stream)
    ctx.check(torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(host["prim"], prim.cpu().numpy()) and np.array_equal(host["inst"], inst.cpu().numpy())
    assert np.all(same(host["t"], t.cpu().numpy())) and np.all(same(host["bary"], bary.cpu().numpy()))
    hit = host["prim"] >= 0
    triangles = np.array([len(m["indices"].reshape(-1, 3)) for m in sc["meshes"]])
    mesh = np.array([i["mesh"] for i in sc["instances"]])
    assert np.all(host["inst"][hit] < len(mesh)) and np.all(host["inst"][hit] >= 0)
    assert np.all(host["prim"][hit] < triangles[mesh[host["inst"][hit]]])
