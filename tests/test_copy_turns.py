"""The turns of a CTA with bulk copies (cdocker_b200/csrc/copy_turns.cuh) on the CPU: after a wait that
gives up no copy is issued, and the copies in flight land before the CTA leaves its buffer."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_copy_turns_over_a_model_of_the_barrier(tmp_path):
    exe = os.path.join(str(tmp_path), "copy_turns_model")
    subprocess.run([shutil.which("g++") or "g++", "-std=c++14", "-O1", "-Wall", "-Wno-unknown-pragmas",
                    "-I", os.path.join(ROOT, "cdocker_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cxx", "copy_turns_model.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
