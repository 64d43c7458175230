"""Plain scenes (area lights and the ramp, plain materials) have shade kernels of their own. An
unused coated material makes a scene not plain without changing its image, so the same scene
through both kernels must give the same bits: every background, with and without lights and an
environment, through waves, the tail and the batched queue; and the same gradients."""
import copy

import numpy as np
import pytest

from repackshot_b200 import scenes

pytestmark = pytest.mark.gpu


def _knot():
    return scenes.product_scene(width=61, height=37, spp=3, depth=9, seg_u=64, seg_v=32)


def _varied(make, **fields):
    s = make()
    for k, v in fields.items():
        setattr(s, k, v)
    s.width, s.height = 61, 37
    return s


def _general(s):
    g = copy.deepcopy(s)
    g.materials.append(scenes.Material(coat=1.0, coat_roughness=0.3))
    return g


def _film(scene, spp):
    film = scene.film()
    film.render(0, spp)
    return film.read()


CASES = [
    lambda: _knot(),
    lambda: _varied(_knot, background_mode=1, clamp_indirect=0.5),
    lambda: _varied(_knot, background_mode=2, lights=[]),
    lambda: _varied(_knot, env_strength=0.0, max_depth=2),
    lambda: _varied(_knot, env_strength=0.0, lights=[]),
    lambda: _varied(scenes.example_scene, pixel_filter=3, edge_supersample=2),
    lambda: _varied(scenes.cfg0_scene, max_depth=1),
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("tail", [0, 1 << 14])
def test_plain_equals_general(case, tail):
    import repackshot_b200 as rtg
    s = CASES[case]()
    films = []
    for desc in (s, _general(s)):
        scene = rtg.Scene(scenes.to_rsb(desc))
        scene.set_tuning(tail_paths=tail)
        films.append(_film(scene, 5))
    for a, b in zip(*films):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_plain_queue_and_mixed_queue():
    import repackshot_b200 as rtg
    base = _knot()
    other = copy.deepcopy(base)
    other.width, other.height = 48, 80
    jobs = [base, _general(base), other]
    for chosen in ([base, other], jobs):  # all plain; one general job takes the general kernel for all
        scene = rtg.Scene(scenes.to_rsb(base))
        queue = rtg.Queue(scene)
        films = [queue.add(scenes.to_rsb(j, meshes=False), 0, 3, j.width, j.height) for j in chosen]
        queue.run()
        for j, f in zip(chosen, films):
            want = _film(rtg.Scene(scenes.to_rsb(j)), 3)
            for a, b in zip(f.read(), want):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_plain_gradients():
    import repackshot_b200 as rtg
    s = scenes.adjoint_scene(40, 24, 4, 5)
    target = np.full((24, 40, 3), 0.3, np.float32)
    out = []
    for desc in (s, _general(s)):
        scene = rtg.Scene(scenes.to_rsb(desc))
        loss, grads, _ = scene.adjoint(scene.film(), target, 0, 4)
        out.append((loss, grads))
    (la, ga), (lb, gb) = out
    nm = len(s.materials)
    assert la == lb
    # the same terms summed by atomics in another order: within rounding of their magnitudes
    assert np.allclose(ga[:4 * nm], gb[:4 * nm], rtol=1e-4, atol=1e-7)
    assert np.allclose(ga[4 * nm:], gb[4 * nm + 4:], rtol=1e-4, atol=1e-7)
