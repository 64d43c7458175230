"""The rounds of a wave: the block-wise material sort against unsorted shading, and each round's shadow
rays traced with the next round's extension rays against launches of their own (a timed wave's),
shadow walks included. Each path's arithmetic is its own, so the films have the same bits."""
import copy

import numpy as np
import pytest

from repackshot_b200 import scenes

pytestmark = pytest.mark.gpu


def _many_materials(n):
    """Instances in n materials: keys up to the last one, which all higher materials share."""
    s = scenes.cfg4_scene(depth=4, n_instances=n)
    s.meshes = [scenes.displaced_sphere(200), scenes.floor_quad(0.0, 20000.0, 0)]
    base = s.materials[0]
    s.materials = [copy.copy(base) for _ in range(n)]
    for k, m in enumerate(s.materials):
        m.base_color = (0.2 + 0.6 * (k % 7) / 7, 0.2 + 0.6 * (k % 11) / 11, 0.2 + 0.6 * (k % 5) / 5)
    for k, i in enumerate(s.instances):
        i.material_id = k % n
    return s


def _film(desc, width, height, spp, timed=False, **tuning):
    import repackshot_b200 as rtg
    desc.width, desc.height = width, height
    scene = rtg.Scene(scenes.to_rsb(desc))
    scene.set_tuning(**tuning)
    scene.timing(timed)
    film = scene.film()
    film.render(0, spp)
    return film.read()


# Paths around one and two chunks of 2048 a sort block takes, one warp's and one path's.
SIZES = [(1, 1, 1), (31, 1, 1), (33, 1, 1), (89, 23, 1), (64, 32, 1), (683, 3, 1), (241, 17, 1), (64, 64, 3)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("materials", [3, 255, 300])
def test_material_sort_keeps_the_bits(size, materials):
    films = [_film(_many_materials(materials), *size, material_sort=on, tail_paths=0) for on in (True, False)]
    for a, b in zip(*films):
        assert np.array_equal(a, b)


SHADOWS = {"plain": lambda: scenes.product_scene(spp=3, depth=9, seg_u=64, seg_v=32), "cut-outs and thin walls": scenes.e5_scene,
           "light kinds": scenes.light_kinds_scene}


@pytest.mark.parametrize("name", list(SHADOWS))
@pytest.mark.parametrize("size", [(1, 1, 1), (33, 7, 5), (96, 64, 4)])
@pytest.mark.parametrize("tail", [0, 1 << 14])
def test_shadow_rays_together_and_apart_have_the_same_bits(name, size, tail):
    films = [_film(SHADOWS[name](), *size, timed=timed, tail_paths=tail) for timed in (False, True)]
    for a, b in zip(*films):
        assert np.array_equal(a, b)


# One path, a warp less and more than full, and more paths than all pairs of warps hold at once.
@pytest.mark.parametrize("name", ["plain", "light kinds"])
@pytest.mark.parametrize("size", [(1, 1, 1), (31, 1, 1), (65, 1, 1), (67, 41, 3), (160, 120, 3)])
def test_the_tail_has_the_wavefronts_bits(name, size):
    films = [_film(SHADOWS[name](), *size, tail_paths=tail) for tail in (0, 1 << 20)]
    for a, b in zip(*films):
        assert np.array_equal(a, b)
