"""Host code of the library against a CUDA runtime without a GPU
(tests/cpp/fake_cudart.h): what a call has set up, and what it leaves in flight,
which on a device only a failing or an unlucky run would show."""
import glob
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.parametrize("name", ["test_noalloc_setup", "test_nothing_in_flight", "test_host_pages", "test_server_output"])
def test_host_code(built, tmp_path, name):
    objects = sorted(glob.glob(os.path.join(ROOT, "texpresso_gb300", "_build", "*.o")))
    cuda = os.path.join(os.path.dirname(os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")), "..", "include")
    if not objects or not os.path.isdir(cuda):
        pytest.skip("needs the library's object files and the CUDA headers")
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", cuda, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", name + ".cpp")] + objects + ["-lpthread", "-ldl", "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
