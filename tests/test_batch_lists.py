"""Memory that runs out while a job's batches are sorted into their lists, on
several threads, reaches the caller as an exception instead of ending the
process."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("where", ["helpers", "caller"])
def test_out_of_memory_in_batch_lists(sbp, tmp_path, where):
    from gsap_b200 import build
    exe = tmp_path / "batch_lists"
    lib = os.path.join(ROOT, "gsap_b200")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(lib, "csrc"), "-I", cuda,
                    os.path.join(ROOT, "tests", "batch_lists_main.cpp"),
                    os.path.join(lib, "libsbp.so"), f"-Wl,-rpath,{lib}", "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe), where], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
