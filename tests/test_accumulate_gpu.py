"""Images from the radiance planes and shading records from the vertex arrays:
the image is the running mean, in sample order, of the samples the sample call
gives (bit for bit, at sample counts around the eight that the kernel loads
ahead, in one chunk, several, and a batch), and a mesh without normals or uvs
renders as one with zeros."""
import numpy as np
import pytest

import tpt
import tpt_scenes

pytestmark = pytest.mark.gpu


def running_mean(samples, exposure):
    """main.rs:107-123 in float32: mean += (x - mean) / (k + 1), times exposure."""
    mean = np.zeros(samples.shape[0:1] + (3,), np.float32)
    for k in range(samples.shape[1]):
        mean = mean + (samples[:, k] - mean) / np.float32(k + 1)
    return mean * np.float32(exposure)


@pytest.mark.parametrize("spp", [1, 2, 7, 8, 9, 16, 17, 41])
@pytest.mark.parametrize("capacity", [0, 1024])
def test_image_is_the_running_mean_of_its_samples(ctx, spp, capacity):
    import torch

    w, h = 37, 23
    sc = tpt_scenes.cornell_box(3, tpt_scenes.LAMBERT)
    sc["camera"] = dict(sc["camera"], exposure=1.7)
    s = tpt.Scene(ctx, sc["meshes"], sc["instances"], materials=sc["materials"])
    job = s.job(sc["camera"], w, h, spp, 3)
    stream = torch.cuda.current_stream().cuda_stream
    samples = torch.empty((w * h, spp, 3), device="cuda")
    s.render_samples_device(job, 0, w * h * spp, samples.data_ptr(), stream)
    images = [torch.empty((w * h, 3), device="cuda") for _ in range(3)]
    try:
        ctx.wavefront_capacity = capacity
        s.render_device(job, images[0].data_ptr(), stream)
        ctx.render_batch_device([job, job], [im.data_ptr() for im in images[1:]], stream)
        torch.cuda.synchronize()
    finally:
        ctx.wavefront_capacity = 0  # the default
    want = running_mean(samples.cpu().numpy(), 1.7)
    for im in images:
        assert np.array_equal(im.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("n_meshes", [1, 2, 9])
def test_missing_attributes_are_zeros(ctx, n_meshes):
    rng = np.random.default_rng(n_meshes)
    bare, zeros, instances = [], [], []
    for k in range(n_meshes):
        tris = int(rng.integers(1, 40))
        p = rng.uniform(-1, 1, (3 * tris, 3)).astype(np.float32)
        idx = rng.permutation(3 * tris).astype(np.uint32)
        bare.append({"positions": p, "indices": idx})
        zeros.append({"positions": p, "indices": idx, "normals": np.zeros_like(p),
                      "uvs": np.zeros((3 * tris, 2), np.float32)})
        instances.append(tpt_scenes.identity_instance(k, k % 2))
    mats = [{"kind": tpt_scenes.LAMBERT, "rho": np.full(3, 0.6, np.float32)},
            {"kind": tpt_scenes.EMISSIVE, "color": np.ones(3, np.float32), "strength": np.float32(2.0)}]
    cam = {"eye": (0.0, 0.0, 4.0), "look_at": (0.0, 0.0, 0.0), "up": (0.0, 1.0, 0.0), "fov_y": 0.6, "exposure": 1.0}
    a, b = (tpt.Scene(ctx, m, instances, materials=mats).render(cam, 48, 40, 8, 4) for m in (bare, zeros))
    assert np.array_equal(a, b)
    assert n_meshes == 1 or a.max() > 0
