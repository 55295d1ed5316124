"""A batch step that ends with an error (tests/host_c/batch_step_errors.cu: the
batch code with fakes of the runtime and of the session functions): an input
the runtime refuses leaves every session as it was, a frame that cannot be
launched leaves the frames before it finished and the others as they were,
nothing stays in flight, and the next step runs.  A session made at the address
of a destroyed one is another session to a batch's cached graphs."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_errors(tmp_path):
    nvcc = next((c for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc"))
                 if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc absent")
    exe = tmp_path / "batch_step_errors"
    subprocess.check_call([nvcc, "-std=c++17", "-O0", "-w", "-cudart", "none", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-I", os.path.join(HERE, "..", "include"), "-o", str(exe),
                           os.path.join(HERE, "host_c", "batch_step_errors.cu"),
                           os.path.join(HERE, "host_c", "fake_cudart.cpp")])
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=120).stdout
    rows = {line.split()[0]: [int(v) for v in line.split()[1:]] for line in out.splitlines()}
    assert set(rows) == {"refused_input", "failed_launch", "other_modes", "same_address"}, out
    for name, (runs, failures) in rows.items():
        assert runs > 0 and failures == 0, (name, runs, failures)
