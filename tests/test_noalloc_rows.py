"""The index arithmetic of the no-allocation call's row batches, walked on the CPU."""
import subprocess

from conftest import ROOT


def test_batches_of_rows_stay_inside_what_they_stage(tmp_path):
    exe = tmp_path / "noalloc_batches"
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", str(ROOT / "tests" / "cpp" / "noalloc_batches.cpp"), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout == "ok\n", res.stdout
