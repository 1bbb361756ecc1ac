"""Large copies between device and pageable host memory go on with fewer threads, or one plain copy, where threads or pinned
slots cannot be had: they sit behind a C interface, which must not end the process for want of a thread."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def tool(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host_copy") / "copy_threads")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "glades-ml_b200", "csrc"), "-I", os.path.join(CUDA, "include"),
                    os.path.join(ROOT, "tests", "host", "copy_threads.cpp"), "-o", exe, "-lpthread", "-ldl"], check=True)
    return exe


@pytest.mark.parametrize("threads,slots", [(0, 12), (1, 12), (3, 12), (100, 100), (100, 0), (100, 1), (2, 4)])
def test_copy_goes_on_with_what_can_be_had(tool, threads, slots):
    r = subprocess.run([tool, str(threads), str(slots)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, "status %d\n%s%s" % (r.returncode, r.stdout, r.stderr)
