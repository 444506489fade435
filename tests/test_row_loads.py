"""The rows that the query's tuner samples are read within the caller's array (CPU)."""
import os
import subprocess

from pbig_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_loads_of_a_row_stay_in_the_array(tmp_path):
    exe = str(tmp_path / "row_loads")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", build.CSRC, "-I", os.path.join(build.CUDA_HOME, "include"),
                    os.path.join(HERE, "clients", "row_loads.cc"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
