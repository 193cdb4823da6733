"""A failed product stops Adam within the epoch that it fails in
(tests/cpp/mlp_error_check.cpp)."""
import os
import re
import subprocess

import pytest

import cbmtest

pytestmark = pytest.mark.gpu


def test_training_stops_at_a_failed_product(tmp_path):
    import cerebellum_simulation_b200 as cbm
    libdir = os.path.dirname(cbm.LIB_PATH)
    exe = str(tmp_path / "mlp_error_check")
    cudart = re.search(r"libcudart\S* => (\S+)", subprocess.run(["ldd", cbm.LIB_PATH], check=True, capture_output=True,
                                                                text=True).stdout).group(1)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-I", os.path.join(cbmtest.ROOT, "include"),
                    os.path.join(cbmtest.ROOT, "tests", "cpp", "mlp_error_check.cpp"), "-rdynamic", "-L", libdir,
                    "-lcbm_b200", cudart, "-ldl", f"-Wl,-rpath,{libdir}", "-o", exe], check=True, capture_output=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
