"""Ray queries where the node ranking, the triangle pairs and the split stack can
go wrong: children at equal distances (coincident triangles and instances),
meshes of odd triangle counts (a pair holds triangles of two meshes), and
stacks on both sides of the shared-memory part's 12 entries."""
import numpy as np
import pytest

import tpt
import tpt_scenes
from test_device_errors_gpu import deep_chain_qbvh, rays_down_the_chain
from test_traverse_gpu import assert_same, build_both, instance_from

pytestmark = pytest.mark.gpu


def coincident_mesh(n, rng):
    """n triangles, every second one a copy of the one before."""
    p = rng.uniform(-1, 1, ((n + 1) // 2, 3, 3)).astype(np.float32)
    p = np.repeat(p, 2, axis=0)[:n]
    return {"positions": p.reshape(-1, 3), "indices": np.arange(3 * n, dtype=np.uint32)}


@pytest.mark.parametrize("counts", [(1,), (2, 1), (3, 5, 7), (1, 1, 1, 9), (31, 17, 2)])
def test_coincident_triangles_and_odd_meshes(ctx, counts):
    rng = np.random.default_rng(len(counts))
    meshes = [coincident_mesh(n, rng) for n in counts]
    instances = []
    for i in range(12):
        l2w = np.eye(4)
        l2w[:3, 3] = np.round(rng.uniform(-2, 2, 3))
        instances += [instance_from(i % len(meshes), l2w)] * (1 + i % 2)  # some instances twice
    g, s = build_both(ctx, meshes, instances)
    rays = tpt_scenes.incoherent_rays(1 << 14, seed=5, cube=8.0)
    rays[0:3] -= 4.0
    rays[0:3, ::4] = np.round(rays[0:3, ::4])
    for mode in (tpt.CLOSEST_HIT, tpt.ANY_HIT):
        ref = g.query(rays, mode)
        dev = s.closest_hit(rays, mode, want_instance=True, want_bary=True)
        assert_same(dev, ref, "mode %d" % mode)
        hit = ref["prim"] >= 0
        assert hit.any()
        assert np.array_equal(dev["inst"], ref["inst"])
        assert np.array_equal(dev["bary"][:, hit].view(np.uint32), ref["bary"][:, hit].view(np.uint32))


@pytest.mark.parametrize("levels", [1, 10, 11, 12, 13, 14, 60, 126])
def test_stack_depths_around_the_shared_part(ctx, levels):
    tri = {"positions": np.array([[-1, -1, 50], [1, -1, 50], [0, 1, 50]], np.float32),
           "indices": np.array([0, 1, 2], np.uint32)}
    g, _ = build_both(ctx, [tri], [tpt_scenes.identity_instance()])
    s = tpt.Scene(ctx, [dict(tri, qbvh=deep_chain_qbvh(levels))], [tpt_scenes.identity_instance()])
    rays = rays_down_the_chain(256)
    ref = g.query(rays, 0)
    assert (ref["prim"] == 0).all()
    assert_same(s.closest_hit(rays), ref, "%d levels" % levels)
