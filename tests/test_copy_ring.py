"""A wait for a bulk copy that runs out: nothing more is asked for on a barrier whose copy is still in flight, and the copies in
flight are waited for before the block ends.  The kernels' sequences on made-up barriers, no GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_copy_is_asked_for_behind_a_wait_that_ran_out(tmp_path):
    exe = str(tmp_path / "copy_ring")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "glades-ml_b200", "csrc"),
                    os.path.join(ROOT, "tests", "host", "copy_ring.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
