"""The device traversal, built for the host, against the oracle's: its slab test passes boxes by
rounded planes and leaves the ends of the interval to each leaf's exact box, so it must give the
reference's hits for every kind of ray (incoherent, along the axes, leaving surfaces, short, with
tiny directions, with a negative t_min) and every kind of tree (one world-space tree, two levels,
single leaves, flat boxes)."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from rays import edge_rays, random_rays, surface_rays
from repackshot_b200 import build, scenes

LO, HI = (-1500, -1500, 0), (1500, 1500, 2500)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    objs = [str(build.OBJ / f"{n}.cpp.o") for n in ("rtg_scene", "rtg_section", "rtg_bitmap", "rtg_ies", "rtg_tables", "rtg_energy")]
    if not all(Path(o).exists() for o in objs):
        build.build()
    lib = tmp_path_factory.mktemp("host") / "trace_host.so"
    subprocess.run([build.CXX, "-O2", "-std=c++17", "-fPIC", "-ffp-contract=off", f"-I{build.CUDA_HOME}/include", "-shared",
                    str(Path(__file__).parent / "trace_host.cpp"), *objs, "-o", str(lib), "-lpthread"], check=True)
    L = ctypes.CDLL(str(lib))
    L.host_load.restype = ctypes.c_void_p
    L.host_load.argtypes = [ctypes.c_char_p, ctypes.c_uint64]
    L.host_free.argtypes = [ctypes.c_void_p]
    L.host_trace.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    return L


def _instances():
    return scenes.cfg4_scene(width=64, height=64, n_instances=60)


def _knot():
    return scenes.product_scene(width=96, height=64, spp=4, depth=12, seg_u=64, seg_v=32)


@pytest.mark.parametrize("make", [scenes.cfg0_scene, scenes.example_scene, scenes.e5_scene, scenes.emissive_scene, _knot, _instances, scenes.sun_triangle_scene])
def test_traversal_equals_oracle(host, oracle_lib, make):
    rsb = scenes.to_rsb(make())
    ref = oracle_lib.OracleScene(rsb)
    handle = host.host_load(rsb, len(rsb))
    assert handle
    short = random_rays(2000, LO, HI, seed=8)
    short[:, 7] = np.random.default_rng(1).random(len(short)) * 1000
    axis = random_rays(2000, LO, HI, seed=11)
    axis[:, 3:6] = np.eye(3)[np.arange(2000) % 3] * np.where(np.arange(2000) % 2, 1, -1)[:, None]
    axis[::5, 0:3] = np.round(axis[::5, 0:3] / 100) * 100
    behind = random_rays(2000, LO, HI, seed=12)
    behind[:, 6] = -500
    tiny = random_rays(2000, LO, HI, seed=13)
    tiny[:, 3:6] *= np.float32(1e-6)
    tiny[:, 6] = 1
    for rays in (random_rays(4000, LO, HI, seed=5), edge_rays(), surface_rays(ref, 4000, 9), short, axis, behind, tiny):
        rays = np.ascontiguousarray(rays, np.float32)
        for camera in (0, 1):
            want, _ = ref.trace(rays, camera=bool(camera))
            forms = (0, 1) if (rays[:, 6] > 0).all() else (0,)
            for positive in forms:
                got = np.zeros((len(rays), 3), np.uint32)
                assert host.host_trace(handle, rays.ctypes.data, len(rays), 0, camera, positive, got.ctypes.data) == 0
                assert np.array_equal(got, want)
                flags = np.zeros(len(rays), np.uint32)
                assert host.host_trace(handle, rays.ctypes.data, len(rays), 1, camera, positive, flags.ctypes.data) == 0
                assert np.array_equal(flags != 0, want[:, 0] != 0xFFFFFFFF)
    host.host_free(handle)
