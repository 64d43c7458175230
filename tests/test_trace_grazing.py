"""Rays that graze a flat mesh, on the device traversal built for the host: there the triangle test's t
is off by far more than any fixed part of a box, so the tree may leave out no triangle whose leaf the
reference looks into. Flat grids of 1 to 10,000 units turned any way, as one world-space tree and as
an instance of a two-level one, against the oracle."""
import numpy as np
import pytest

from repackshot_b200 import scenes
from test_trace_host import host  # noqa: F401 (the fixture)


def flat_grid(g, n, size, jitter):
    x = np.linspace(-size / 2, size / 2, n + 1)
    p = np.stack(np.meshgrid(x, x, indexing="ij"), -1).reshape(-1, 2)
    p = np.concatenate([p + (g.random(p.shape) - 0.5) * jitter * size / n, np.zeros((len(p), 1))], 1)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = i * (n + 1) + j
    index = np.stack([a, a + n + 1, a + 1, a + 1, a + n + 1, a + n + 2], -1).reshape(-1).astype(np.uint32)
    return scenes.Mesh(p.astype(np.float32), np.zeros((len(p), 3), np.float32), index)


def grazing_rays(g, n, size, turn, move):
    """Through points of the grid, 1e-8 to 1e-2 off its plane, some right in it, some along its axis."""
    at = np.concatenate([(g.random((n, 2)) - 0.5) * size, np.zeros((n, 1))], 1)
    angle = g.random(n) * 2 * np.pi
    d = np.stack([np.cos(angle), np.sin(angle), 10.0 ** g.uniform(-8, -2, n) * g.choice([-1, 1], n)], -1)
    d[::4, 2] = 0
    d[1::4, 0] = np.sign(d[1::4, 0])
    d[1::4, 1] = 0
    o = at - d * (size * 10.0 ** g.uniform(-1, 0.5, n))[:, None]
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 3:6], rays[:, 6], rays[:, 7] = o @ turn.T + move, d @ turn.T, 1e-3, np.inf
    return rays


@pytest.mark.parametrize("instanced", [False, True])
@pytest.mark.parametrize("seed", range(12))
def test_grazing_rays_equal_oracle(host, oracle_lib, instanced, seed):  # noqa: F811
    g = np.random.default_rng(seed)
    size = 10.0 ** g.uniform(0, 4)
    mesh = flat_grid(g, int(g.integers(8, 60)), size, 0.5 * (seed % 2))
    turn, _ = np.linalg.qr(g.normal(size=(3, 3)))
    turn *= np.linalg.det(turn)
    move = g.normal(size=3) * size
    rays = grazing_rays(g, 8000, size, turn, move)
    instances = [scenes.Instance(0)]
    meshes = [mesh]
    if instanced:
        instances = [scenes.Instance(0, rows=tuple(float(v) for r in range(3) for v in (*turn[r], move[r]))), scenes.Instance(1)]
        meshes.append(scenes.floor_quad(-20 * size, 10 * size, 0))
    else:
        mesh.positions = (mesh.positions.astype(np.float64) @ turn.T + move).astype(np.float32)
    rsb = scenes.to_rsb(scenes.Scene(materials=[scenes.Material()], meshes=meshes, instances=instances, width=8, height=8))
    ref = oracle_lib.OracleScene(rsb)
    handle = host.host_load(rsb, len(rsb))
    assert handle
    want, _ = ref.trace(rays)
    assert (want[:, 0] == 0).sum() > 1000
    got = np.zeros((len(rays), 3), np.uint32)
    assert host.host_trace(handle, rays.ctypes.data, len(rays), 0, 0, 1, got.ctypes.data) == 0
    flags = np.zeros(len(rays), np.uint32)
    assert host.host_trace(handle, rays.ctypes.data, len(rays), 1, 0, 1, flags.ctypes.data) == 0
    host.host_free(handle)
    assert np.array_equal(got, want)
    assert np.array_equal(flags, ref.occluded(rays))
