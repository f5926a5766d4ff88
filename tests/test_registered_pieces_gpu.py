"""Host queries on memory that was page-locked in pieces or in part: the planes of
the rays and results are separate registrations, or some of them pageable."""
import ctypes as C
import mmap

import numpy as np
import pytest

import tpt
import tpt_scenes

pytestmark = pytest.mark.gpu


class Planes:
    """k planes of n floats in anonymous pages, the named ranges of planes page-locked."""

    def __init__(self, k, n, pieces):
        import torch

        self.a = np.frombuffer(mmap.mmap(-1, 4 * k * n), np.float32).reshape(k, n)
        self.rt = torch.cuda.cudart()
        self.locked = []
        for b, e in pieces:
            assert int(self.rt.cudaHostRegister(self.a[b].ctypes.data, 4 * n * (e - b), 0)) == 0
            self.locked.append(self.a[b].ctypes.data)

    def __enter__(self):
        return self

    def __exit__(self, *_):
        for p in self.locked:
            self.rt.cudaHostUnregister(p)


@pytest.mark.parametrize("n", [1024, 204800])  # whole pages a plane; one chunk and four
@pytest.mark.parametrize("rays_locked", [[(k, k + 1) for k in range(7)], [(0, 3), (3, 7)], [(0, 1)], []],
                         ids=["planes", "two", "first", "none"])
@pytest.mark.parametrize("out_locked", [[(k, k + 1) for k in range(6)], [(0, 2), (2, 4)], []],
                         ids=["planes", "some", "none"])
def test_rays_and_results_locked_in_pieces(ctx, n, rays_locked, out_locked):
    import torch

    torch.zeros(1, device="cuda")
    s = tpt.Scene(ctx, [tpt_scenes.sphere_soup(3, 64, 12.0)], [tpt_scenes.identity_instance()])
    with Planes(7, n, rays_locked) as rays, Planes(6, n, out_locked) as out:  # prim, t, instance, three of bary
        rays.a[:] = tpt_scenes.incoherent_rays(n, seed=n, cube=12.0)
        rays.a[6] = 9.0
        for mode in (tpt.CLOSEST_HIT, tpt.ANY_HIT):
            want = s.closest_hit(np.array(rays.a), mode, want_instance=True, want_bary=True)
            out.a[:] = -7.0
            st = tpt.lib().tpt_traverse(ctx.h, s.h, C.c_void_p(rays.a.ctypes.data), n, mode,
                                        *[C.c_void_p(out.a[k].ctypes.data) for k in range(4)])
            assert st == 0
            got = out.a.view(np.uint32)
            assert np.array_equal(got[0], want["prim"].view(np.uint32)) and (want["prim"] >= 0).any()
            assert np.array_equal(got[1], want["t"].view(np.uint32))
            assert np.array_equal(got[2], want["inst"].view(np.uint32))
            assert np.array_equal(got[3:], want["bary"].view(np.uint32))
