"""disco_b200_plan_execute with no host memory left: a C++ program whose operator
new throws during the call.  The call, which used to allocate nothing, sums by the
plain kernel then; an exception through the C entry would end the program."""
import os
import shutil
import subprocess

import pytest

from disco_b200 import _capi as C

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_execute_without_host_memory(tmp_path):
    cxx = os.environ.get("DISCO_CXX", "g++")
    if shutil.which(cxx) is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "no_memory_driver"
    subprocess.run([cxx, "-std=c++14", "-O2", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(CUDA, "include"),
                    os.path.join(ROOT, "tests", "cpp", "no_memory_driver.cpp"), "-L", C.LIB_DIR, "-ldisco_b200",
                    "-L", os.path.join(CUDA, "lib64"), "-lcudart", f"-Wl,-rpath,{C.LIB_DIR}",
                    f"-Wl,-rpath,{os.path.join(CUDA, 'lib64')}", "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    without, with_memory, diff, most = r.stdout.split()
    assert (int(without), int(with_memory)) == (C.DISCO_OK, C.DISCO_OK)
    assert float(most) > 0.1 and float(diff) <= 2e-14 * 2 + 2e-14        # plain against cells, as in test_tree_gpu.py
