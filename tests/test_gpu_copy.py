"""Copies of a film's planes and of the denoiser's: staged through pinned memory by several threads from
4 MiB on, in pieces of 1 MiB a plane. Into (and out of) memory that is pinned already they are plain
copies, so both must give the same bytes."""
import ctypes

import numpy as np
import pytest

from repackshot_b200 import scenes

pytestmark = pytest.mark.gpu


def _pinned(shape):
    import torch
    return torch.zeros(shape, dtype=torch.float32).pin_memory().numpy()


def _planes(film, make):
    import repackshot_b200 as rtg
    out = [make((film.h, film.w, 3))] + [make((film.h, film.w)) for _ in range(3)]
    for a in out:
        a.fill(np.float32(-7))
    assert rtg.lib().rtg_film_read(film.handle, *(a.ctypes.data_as(ctypes.c_void_p) for a in out)) == 0
    return out


# Under and just over 4 MiB, whole pieces, ragged ones, and more than the threads' slots at once.
@pytest.mark.parametrize("size", [(418, 418), (419, 418), (512, 512), (613, 997), (1280, 720)])
def test_film_planes_arrive_whole(size):
    import repackshot_b200 as rtg
    s = scenes.product_scene(width=size[0], height=size[1], spp=1, depth=2, seg_u=64, seg_v=32)
    film = rtg.Scene(scenes.to_rsb(s)).film()
    film.render(0, 1)
    for a, b in zip(_planes(film, lambda shape: np.zeros(shape, np.float32)), _planes(film, _pinned)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("size", [(16, 16), (280, 267), (281, 270), (640, 367)])
def test_denoised_planes_arrive_whole(size):
    import repackshot_b200 as rtg
    n = size[0] * size[1]
    g = np.random.default_rng(n)
    planes = g.random(14 * n, dtype=np.float32)
    planes[12 * n:].view(np.uint32)[:] = 1  # part and material
    pinned = _pinned(14 * n)
    pinned[:] = planes
    for _ in range(2):  # the second call on the device block that the first one left
        a = rtg.denoise(planes.view(np.uint32), *size, 16)
        out = _pinned(4 * n)
        assert rtg.lib().rtg_denoise_with(0, ctypes.c_float(1.0), size[0], size[1], 0, size[1], 16, 0, size[1],
                                          pinned.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p)) == 0
        assert np.array_equal(a, out)
