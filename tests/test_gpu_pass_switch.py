"""Switching the GR pass in mid-run, to every kind and tiling and with spikes in
flight, changes no result; neither does a switch that fails at any of its
allocations, after which the pass before it goes on (tests/cpp/pass_switch_check.cpp)."""
import os
import re
import subprocess

import pytest

import cbmtest

pytestmark = pytest.mark.gpu


def build(dest_dir):
    import cerebellum_simulation_b200 as cbm
    libdir = os.path.dirname(cbm.LIB_PATH)
    exe = os.path.join(dest_dir, "pass_switch_check")
    cudart = re.search(r"libcudart\S* => (\S+)", subprocess.run(["ldd", cbm.LIB_PATH], check=True, capture_output=True,
                                                                text=True).stdout).group(1)
    cmd = ["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-I", os.path.join(libdir, "csrc"),
           os.path.join(cbmtest.ROOT, "tests", "cpp", "pass_switch_check.cpp"), "-rdynamic", "-L", libdir, "-lcbm_b200",
           cudart, "-ldl", f"-Wl,-rpath,{libdir}", "-o", exe]
    subprocess.run(cmd, check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("batch", [False, True])
def test_pass_switches_keep_the_network(batch, tmp_path):
    from cerebellum_simulation_b200 import networks
    paths = []
    # networks that every pass kind runs: 131,072 GR, and 262,144
    for i, dims in enumerate(((9, 8, 5, 5, 10), (10, 8, 5, 5, 10))[:1 + batch]):
        st = networks.build_random_network(*dims, networks.act_params("dense"), seed=5 + i, go_out_per_gr=4,
                                           mf_per_go=16, vel=147)
        paths.append(str(tmp_path / f"net{i}.state"))
        st.writeState(paths[-1])
    out = str(tmp_path / "out.txt")
    p = subprocess.run([build(str(tmp_path)), *paths, out], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr
    refused = int(re.search(r"(\d+) refused", open(out).read()).group(1))
    assert refused >= 10
