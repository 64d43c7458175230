"""A scene on a stream of the caller's: an ordinary one, the legacy default stream and
cudaStreamPerThread. Pictures and planes of more than 4 MiB go into pageable memory right after the
kernels that make them; each has the bytes that the library's own stream gives."""
import ctypes

import numpy as np
import pytest

from repackshot_b200 import scenes

pytestmark = pytest.mark.gpu


def _pictures(film):
    out = []
    for ev in (0.0, 1.5, -2.0):  # another picture each time, so that a stale one shows
        out += [film.srgb(ev=ev), film.srgb(ev=ev, bits=16), film.denoise(5, strength=1.0), *film.read()]
    return out


@pytest.mark.parametrize("stream", ["own", "legacy", "per-thread"])
def test_large_reads_follow_the_callers_stream(stream):
    import torch

    import repackshot_b200 as rtg
    scene = rtg.Scene(scenes.to_rsb(scenes.product_scene(width=1920, height=1080, spp=1, depth=2, seg_u=64, seg_v=32)))
    film = scene.film()
    film.fuse_guides()
    film.render(0, 5)
    want = _pictures(film)
    theirs = torch.cuda.Stream()
    handle = {"own": theirs.cuda_stream, "legacy": 1, "per-thread": 2}[stream]
    assert rtg.lib().rtg_set_stream(scene.handle, ctypes.c_void_p(handle)) == 0
    got = _pictures(film)
    assert rtg.lib().rtg_set_stream(scene.handle, None) == 0
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
