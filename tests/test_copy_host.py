"""The staged copies of pageable memory on a CUDA runtime of the host's own (copy_host.cpp): whole bytes
in a stream's order, for an ordinary stream and for cudaStreamPerThread, which names another stream in
each of the copies' threads."""
import subprocess
from pathlib import Path

import pytest

from repackshot_b200 import build


@pytest.fixture(scope="module")
def copies(tmp_path_factory):
    exe = tmp_path_factory.mktemp("copies") / "copy_host"
    subprocess.run([build.CXX, "-O2", "-std=c++17", f"-I{build.CUDA_HOME}/include", str(Path(__file__).parent / "copy_host.cpp"), "-o", str(exe), "-lpthread"],
                   check=True)
    return exe


@pytest.mark.parametrize("mode", ["stream", "per-thread"])
@pytest.mark.parametrize("size", [1000, (4 << 20) - 1, 4 << 20, (9 << 20) + 12345])
def test_copies_arrive_in_the_streams_order(copies, mode, size):
    r = subprocess.run([str(copies), mode, str(size)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "0", (r.returncode, r.stdout, r.stderr)


def test_no_memory_for_the_threads(copies):
    r = subprocess.run([str(copies), "no-memory"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "0", (r.returncode, r.stdout, r.stderr)


def test_another_threads_capture_goes_on(copies):
    r = subprocess.run([str(copies), "captured-elsewhere"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "0", (r.returncode, r.stdout, r.stderr)
