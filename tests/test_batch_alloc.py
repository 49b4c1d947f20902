"""Work space of the batched Jacobian products when memory runs short, with an allocator of the test's own on the CPU
(batch_alloc_check.cpp): all buffers of a batch or none, the batch halved until it fits."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_all_buffers_of_a_batch_or_none(tmp_path):
    exe = str(tmp_path / "batch_alloc_check")
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Wextra", "-Werror",
                        "-I" + os.path.join(os.path.dirname(HERE), "dpgsolver_gb300", "csrc"), "-o", exe,
                        os.path.join(HERE, "batch_alloc_check.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "all checks passed" in r.stdout, r.stdout
