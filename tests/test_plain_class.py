"""Which scenes are plain (and take the shade kernels of their own): those that test_gpu_plain.py compares
are, their general versions are not, nor is a scene with any one of the things that plain kernels leave
out."""
import copy
import ctypes
import subprocess
from pathlib import Path

import pytest

from repackshot_b200 import build, scenes
from test_gpu_plain import CASES, _general, _knot


@pytest.fixture(scope="module")
def plain(tmp_path_factory):
    build.build()
    objs = [str(build.OBJ / f"{n}.cpp.o") for n in ("rtg_scene", "rtg_section", "rtg_bitmap", "rtg_ies", "rtg_tables", "rtg_energy")]
    lib = tmp_path_factory.mktemp("scene") / "scene_host.so"
    subprocess.run([build.CXX, "-O2", "-std=c++17", "-fPIC", "-ffp-contract=off", f"-I{build.CUDA_HOME}/include", "-shared",
                    str(Path(__file__).parent / "scene_host.cpp"), *objs, "-o", str(lib), "-lpthread"], check=True)
    f = ctypes.CDLL(str(lib)).host_plain
    f.argtypes = [ctypes.c_char_p, ctypes.c_uint64]
    f.restype = ctypes.c_uint32

    def of(s):
        rsb = scenes.to_rsb(s)
        return f(rsb, len(rsb))
    return of


@pytest.mark.parametrize("case", range(len(CASES)))
def test_compared_scenes_are_plain_and_general(plain, case):
    s = CASES[case]()
    assert plain(s) == 1
    assert plain(_general(s)) == 0


def _with_light(kind):
    def change(s):
        s.lights.append(scenes.Light(kind, (0.0, 0.0, 3000.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0), 10.0, 10.0, (1.0, 1.0, 1.0), 5.0))
    return change


def _with_material(**fields):
    def change(s):
        s.materials[0] = scenes.Material(**fields)
    return change


def _with(**fields):
    def change(s):
        for k, v in fields.items():
            setattr(s, k, v)
    return change


def _with_map(use):
    def change(s):
        s.bitmaps = copy.deepcopy(scenes.e5_scene().bitmaps)
        use(s)
    return change


CHANGES = {
    "sun": _with_light(scenes.LIGHT_SUN), "point": _with_light(scenes.LIGHT_POINT), "spot": _with_light(scenes.LIGHT_SPOT),
    "sky": _with(env_kind=2), "hdri": _with_map(lambda s: _with(env_kind=3, hdri_map=0)(s)),
    "backplate": _with_map(lambda s: _with(background_mode=3, backplate_map=0)(s)),
    "coat": _with_material(coat=0.5), "anisotropy": _with_material(anisotropy=0.3, metallic=1.0), "cut-out": _with_material(opacity=0.5),
    "thin": _with_material(transmission=1.0, flags=scenes.MATERIAL_FLAG_THIN), "no refraction": _with_material(transmission=1.0, ior=1.0),
    "absorption": _with_material(base_color=(0.9, 0.5, 0.5), transmission=1.0, absorption_mm=10.0),
    "emissive": _with_material(kind=scenes.MATERIAL_EMISSIVE, emission=(1.0, 1.0, 1.0), emission_power=1.0),
    "floor": _with(floor_mode=1), "section": _with(section=(1, 0.0, 0.0, 1.0, 500.0)),
}


@pytest.mark.parametrize("name", list(CHANGES))
def test_one_other_thing_makes_a_scene_general(plain, name):
    s = copy.deepcopy(_knot())
    assert plain(s) == 1
    CHANGES[name](s)
    assert plain(s) == 0
