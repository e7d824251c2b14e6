"""The page-locked staging of results on the CPU, with no device: the library's
own Staging (scx_b200/csrc/staging.h) over fakes of its CUDA calls
(tests/cpp/staging_fakes.cpp).  Results come back whether page-locked memory is
granted or refused, a refusal leaves no error behind for a later call, buffers
are used again, and the list keeps no more than its bound."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = ROOT / "tests" / "cpp" / "staging_fakes.cpp"


@pytest.fixture(scope="module")
def fakes(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = Path(nvcc).resolve().parent.parent / "include"
    if cxx is None or not (include / "cuda_runtime_api.h").exists():
        pytest.skip("no C++ compiler or no CUDA headers")
    out = tmp_path_factory.mktemp("staging") / "staging_fakes"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", str(ROOT / "scx_b200" / "csrc"), "-I", str(include), str(SRC),
                    "-o", str(out), "-pthread"], check=True)
    return out


@pytest.mark.parametrize("granted,sizes,want", [
    (99, (100, 70_000, 100), dict(asked=2, freed=0, waits=4, held=(1 << 16) + (1 << 17))),  # used again
    (0, (100, 70_000), dict(asked=3, freed=0, waits=3, held=0)),                             # always refused
    (1, (100, 70_000, 100), dict(asked=2, freed=0, waits=4, held=1 << 16)),                  # refused once
    (99, ((64 << 20) + 1, 100), dict(asked=2, freed=1, waits=3, held=1 << 16)),              # more than is kept
])
def test_results_come_back(fakes, granted, sizes, want):
    r = subprocess.run([str(fakes), str(granted), *map(str, sizes)], capture_output=True, text=True, check=True)
    got = dict((k, int(v)) for k, v in (f.split("=") for f in r.stdout.split()))
    assert got == dict(same=1, error=0, **want)
