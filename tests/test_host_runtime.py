"""The engine's host code against a CUDA runtime without a device (host/fake_cudart.cpp): the order of
operations across streams, the sizes of the buffers that launches and copies get, and the states that failed
allocations and refused adaptations leave.  No GPU."""
import glob
import importlib.util
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "jp-solver_gb300")
HOST = os.path.join(ROOT, "tests", "host")
CUDA = "/usr/local/cuda"


@pytest.fixture(scope="session")
def checks(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(CUDA + "/bin/nvcc"):
        pytest.skip("needs g++ and nvcc")
    spec = importlib.util.spec_from_file_location("jp_engine_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    build.build_lib(verbose=False)
    exe = str(tmp_path_factory.mktemp("host") / "runtime_checks")
    cmd = ["g++", "-std=c++17", "-O1", "-I", CUDA + "/include", "-I", os.path.join(ROOT, "include"), "-I",
           os.path.join(PKG, "csrc"), "-I", HOST]
    cmd += sorted(glob.glob(os.path.join(HOST, "*.cpp"))) + sorted(glob.glob(os.path.join(PKG, "_build", "*.o")))
    r = subprocess.run(cmd + ["-o", exe, "-lpthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


@pytest.mark.parametrize("name", [
    "regrid_orders_list_counts",
    "growth_out_of_memory_then_diag",
    "diag_buffer_of_the_grid",
    "refused_level2_growth_leaves_no_grid",
    "chosen_mapping_takes_every_step",
    "coefficients_search_both_neighbours",
    "in_place_conversions_keep_no_memory",
    "conversions_without_memory",
    "failed_conversion_waits_for_its_copies",
    "replayed_steps_count_their_kernels",
    "upload_precedes_replay_on_its_stream",
    "graphs_order_kernels_as_streams_do",
    "failed_load_leaves_no_grid",
])
def test_host_code(checks, name, tmp_path):
    r = subprocess.run([checks, name], capture_output=True, text=True, timeout=120, cwd=tmp_path)
    assert r.returncode == 0, r.stdout + r.stderr
