"""Scenes whose trees come close to what the traversal stack holds: many instances of a detailed mesh,
and triangles in clusters that grow geometrically. They load, and the device traversal built for the
host has the oracle's hits on them without overflowing its stack."""
import numpy as np
import pytest

from rays import random_rays
from repackshot_b200 import scenes
from test_trace_host import host  # noqa: F401 (the fixture)


def detailed_instances():
    s = scenes.cfg4_scene(width=64, height=64, n_instances=60)
    s.meshes = [scenes.displaced_sphere(399_424), scenes.floor_quad(0.0, 20000.0, 16)]
    return s, (-3000, -3000, 0), (3000, 3000, 2000)


def growing_clusters():
    """8 triangles a cluster, 32 clusters side by side, each four times as large as the one before."""
    g = np.random.default_rng(5)
    p, scale, x = [], 1.0, 0.0
    for _ in range(32):
        c = (g.random((8, 3, 3)) * 0.5 + g.random((8, 1, 3))) * scale
        c[..., 0] += x
        p.append(c.reshape(-1, 3))
        x, scale = x + 2 * scale, scale * 4
    p = np.concatenate(p).astype(np.float32)
    mesh = scenes.Mesh(p, np.zeros_like(p), np.arange(len(p), dtype=np.uint32))
    half = (0.5, 0, 0, 1, 0, 0.5, 0, 0, 0, 0, 0.5, 0)
    s = scenes.Scene(materials=[scenes.Material()], meshes=[mesh, scenes.floor_quad(0.0, 10.0, 0)],
                     instances=[scenes.Instance(0, rows=half), scenes.Instance(1)], width=8, height=8)
    return s, (0, 0, 0), (3000, 1000, 1000)


@pytest.mark.parametrize("make", [detailed_instances, growing_clusters])
def test_deep_trees_load_and_trace(host, oracle_lib, make):  # noqa: F811
    s, lo, hi = make()
    rsb = scenes.to_rsb(s)
    handle = host.host_load(rsb, len(rsb))
    assert handle
    rays = random_rays(2000, lo, hi, seed=3)
    want, _ = oracle_lib.OracleScene(rsb).trace(rays)
    assert (want[:, 0] != 0xFFFFFFFF).sum() > 200
    got = np.zeros((len(rays), 3), np.uint32)
    assert host.host_trace(handle, rays.ctypes.data, len(rays), 0, 0, 1, got.ctypes.data) == 0
    host.host_free(handle)
    assert np.array_equal(got, want)
