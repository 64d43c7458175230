"""rtg_scene_stats counts the triangles that the trees hold: each once in the world-space tree, a shared
mesh's once however often it is placed."""
import pytest

from repackshot_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make,leaf,instanced", [
    (lambda: scenes.Scene(materials=[scenes.Material()], meshes=[scenes.floor_quad(0.0, 10.0, 0)], instances=[scenes.Instance(0)], width=8, height=8), 2, 2),
    (scenes.example_scene, 320 + 2 + 320, 642),
    (lambda: scenes.cfg4_scene(width=64, height=64, n_instances=60), 10_002, 600_002),
])
def test_leaf_triangles(make, leaf, instanced):
    import repackshot_b200 as rtg
    scene = rtg.Scene(scenes.to_rsb(make()))
    assert (scene.leaf_triangles, scene.triangles) == (leaf, instanced)
