"""The per-triangle shading records, gathered on the device at upload, against the
oracle's own vertex arrays: samples of scenes of one, two and nine meshes with
unequal numbers of triangles and vertices, shared vertices, and normals in some
meshes only (a wrong mesh span, index or normal changes a path for good).  Bars of
the Lambert renders' parity test: 99 % of the samples within 1e-5, 99.9 % within
1e-3."""
import numpy as np
import pytest

import oracle as orc
import tpt
import tpt_scenes

CAMERA = {"eye": (0.0, 0.0, 5.0), "look_at": (0.0, 0.0, 0.0), "up": (0.0, 1.0, 0.0), "fov_y": 0.7, "exposure": 1.0}


def mesh(rng, with_normals):
    vertices, triangles = int(rng.integers(8, 40)), int(rng.integers(3, 60))
    m = {"positions": rng.uniform(-1, 1, (vertices, 3)).astype(np.float32),
         "indices": np.concatenate([rng.permutation(vertices)[:3] for _ in range(triangles)]).astype(np.uint32)}
    if with_normals:
        n = np.array([0.0, 0.0, 1.0]) + 0.4 * rng.standard_normal((vertices, 3))
        m["normals"] = (n / np.linalg.norm(n, axis=1, keepdims=True)).astype(np.float32)
    return m


def scene(n_meshes):
    """The meshes side by side, turned and scaled, under a point light."""
    rng = np.random.default_rng(n_meshes)
    side = int(np.ceil(np.sqrt(n_meshes)))
    instances = []
    for k in range(n_meshes):
        q, _ = np.linalg.qr(np.eye(3) + 0.2 * rng.standard_normal((3, 3)))
        l2w = np.eye(4)
        l2w[:3, :3] = q * np.sign(np.diag(q)) * rng.uniform(0.8, 1.1, 3) * 1.6 / side
        l2w[:2, 3] = (np.array([k % side, k // side]) - 0.5 * (side - 1)) * 3.2 / side
        instances.append(tpt_scenes.instance_matrix(k, 0, l2w))
    return {"meshes": [mesh(rng, k % 3 != 1) for k in range(n_meshes)], "instances": instances, "camera": CAMERA,
            "materials": [{"kind": tpt_scenes.LAMBERT, "rho": np.full(3, 0.7, np.float32)}],
            "point_lights": [{"position": (1.0, 2.0, 6.0), "color": (1.0, 0.9, 0.8), "intensity": 400.0}]}


@pytest.mark.gpu
@pytest.mark.parametrize("n_meshes", [1, 2, 9])
def test_samples_match_oracle(ctx, n_meshes):
    import torch

    sc = scene(n_meshes)
    dev = tpt.Scene(ctx, sc["meshes"], sc["instances"], materials=sc["materials"], lights=sc)
    w, h, spp, depth = 48, 40, 8, 5
    n = w * h * spp
    out = torch.empty((n, 3), device="cuda")
    dev.render_samples_device(dev.job(CAMERA, w, h, spp, depth), 0, n, out.data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    d = out.cpu().numpy()
    r = orc.RenderScene(sc, dev.light_tree()).samples(CAMERA, w, h, spp, depth, 0, n)
    rel = np.abs(d - r).max(1) / np.maximum(np.abs(r).max(1), 1e-30)
    assert np.all(np.isfinite(d)) and r.mean() > 0.005
    assert (rel <= 1e-5).mean() >= 0.99, (rel <= 1e-5).mean()
    assert (rel <= 1e-3).mean() >= 0.999, (rel <= 1e-3).mean()
