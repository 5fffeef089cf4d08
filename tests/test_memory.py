"""The device allocator (string_vext_b200/csrc/memory.cu) on a fake CUDA
runtime of host memory (tests/fake_cuda.cpp): refused waits, which no GPU test
brings about, memory given back, and copies from two devices."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not Path(NVCC).exists():
        pytest.skip("needs nvcc")
    out = tmp_path_factory.mktemp("fake") / "fake"
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "-cudart", "none", str(ROOT / "string_vext_b200" / "csrc" / "memory.cu"),
                    str(ROOT / "tests" / "fake_cuda.cpp"), "-o", str(out), "-lpthread"],
                   check=True)
    return out


@pytest.mark.parametrize("scenario", ["refused_wait", "refused_wait_large", "released",
                                      "two_devices", "together"])
def test_allocator(fake, scenario):
    run = subprocess.run([str(fake), scenario], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
