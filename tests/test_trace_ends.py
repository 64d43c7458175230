"""Rays whose interval ends or begins within rounding of a surface (shadow rays to a light flush with a
wall, spans that end on a section's plane), on the device traversal built for the host: a flat box
that begins past t_max or ends before t_min hides its triangles from the reference even where their
computed t lies inside, so hits and misses must be the oracle's, nearest and any, in one tree and in
two levels."""
import numpy as np
import pytest

from rays import random_rays
from repackshot_b200 import scenes
from test_trace_host import LO, HI, _instances, _knot, host  # noqa: F401 (the fixture)


def towards_floor(n, seed):
    rays = random_rays(n, LO, HI, seed=seed)
    to = np.random.default_rng(seed).uniform(-3000, 3000, (n, 3))
    to[:, 2] = 0
    d = to - rays[:, 0:3]
    rays[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return rays


def at_hits(ref, rays, column, seed):
    """The rays that hit, with t_min (6) or t_max (7) at 1 +- 1e-4 ... 1e-7 of the hit, some right there."""
    hits, _ = ref.trace(rays)
    on = hits[:, 0] != 0xFFFFFFFF
    t = hits[on, 2].view(np.float32).astype(np.float64)
    g = np.random.default_rng(seed)
    e = 10.0 ** -g.uniform(4, 7, len(t)) * g.choice([-1, 1], len(t))
    e[::7] = 0
    out = rays[on].copy()
    out[:, column] = (t * (1 + e)).astype(np.float32)
    return out[out[:, 6] > 0]


@pytest.mark.parametrize("make", [scenes.cfg0_scene, scenes.example_scene, scenes.e5_scene, _knot, _instances])
def test_interval_ends_at_a_surface(host, oracle_lib, make):  # noqa: F811
    rsb = scenes.to_rsb(make())
    ref = oracle_lib.OracleScene(rsb)
    handle = host.host_load(rsb, len(rsb))
    assert handle
    for rays in (random_rays(6000, LO, HI, seed=31), towards_floor(6000, 32)):
        for column in (7, 6):
            batch = np.ascontiguousarray(at_hits(ref, rays, column, 33), np.float32)
            assert len(batch) > 500
            want, _ = ref.trace(batch)
            blocked = ref.occluded(batch)
            for positive in (0, 1):
                got = np.zeros((len(batch), 3), np.uint32)
                assert host.host_trace(handle, batch.ctypes.data, len(batch), 0, 0, positive, got.ctypes.data) == 0
                assert np.array_equal(got, want)
                flags = np.zeros(len(batch), np.uint32)
                assert host.host_trace(handle, batch.ctypes.data, len(batch), 1, 0, positive, flags.ctypes.data) == 0
                assert np.array_equal(flags, blocked)
    host.host_free(handle)
