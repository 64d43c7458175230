"""Rays that also look behind their origin (t_min far below zero), on the device traversal built for the
host: the reference visits boxes entered before the origin last, which decides between surfaces that
lie within rounding of each other. Soups of triangles with degenerate and coinciding ones among them,
against the oracle."""
import numpy as np
import pytest

from rays import random_rays
from repackshot_b200 import scenes
from test_trace_host import host  # noqa: F401 (the fixture)


def soup(seed):
    g = np.random.default_rng(seed)
    size = 10 ** (5 * g.random(4)[3] - 2)
    n = int(g.integers(1, 400))
    p = (g.random((n, 1, 3)) - 0.5) * size + (g.random((n, 3, 3)) - 0.5) * size * 10 ** g.uniform(-2, 0)
    kind = g.integers(0, 5, n)
    p[kind == 0, 2] = p[kind == 0, 1]
    p[kind == 1, :, 2] = 0
    p[kind == 2, :, 0] = p[kind == 2, :1, 0]
    p[kind == 3] = np.round(p[kind == 3] / size * 4) * size / 4
    p = p.reshape(-1, 3).astype(np.float32)
    mesh = scenes.Mesh(p, np.zeros_like(p), np.arange(len(p), dtype=np.uint32))
    s = scenes.Scene(materials=[scenes.Material()], meshes=[mesh], instances=[scenes.Instance(0, flags=int(g.integers(0, 2)))], width=8, height=8)
    return s, size


@pytest.mark.parametrize("seed", [3, 40, 98, 116, 175])
def test_rays_from_behind_equal_oracle(host, oracle_lib, seed):  # noqa: F811
    s, size = soup(seed)
    rsb = scenes.to_rsb(s)
    handle = host.host_load(rsb, len(rsb))
    assert handle
    rays = random_rays(4000, (-size,) * 3, (size,) * 3, seed, t_min=-500.0)
    want, _ = oracle_lib.OracleScene(rsb).trace(rays)
    got = np.zeros((len(rays), 3), np.uint32)
    assert host.host_trace(handle, rays.ctypes.data, len(rays), 0, 0, 0, got.ctypes.data) == 0
    host.host_free(handle)
    assert np.array_equal(got, want)
