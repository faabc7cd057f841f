"""The force reduction's scratch when a flag upload fails half way: the
solver's host code over a fake CUDA runtime (fake_cuda_solver.cpp). A scratch
shorter than its list would be written past its end."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def scenario(tmp_path_factory):
    from foil_cfd_gb300 import build_lib
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    exe = tmp_path_factory.mktemp("fake") / "scenario"
    csrc = ROOT / "foil_cfd_gb300" / "csrc"
    # What the scenario does not reach (other launches) stays unresolved.
    subprocess.run(["g++", "-O1", "-std=c++17", "-no-pie", "-I", str(csrc), "-I", str(build_lib._cuda_home() / "include"),
                    str(ROOT / "tests" / "fake_cuda_solver.cpp"), str(csrc / "solver.cpp"),
                    "-Wl,--unresolved-symbols=ignore-all", "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("what", ["grow", "tables", "memset"])
def test_scratch_fits_its_list_after_a_failed_upload(scenario, what):
    r = subprocess.run([str(scenario), what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
