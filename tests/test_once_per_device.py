"""The table that remembers which kernels were allowed their shared memory on which device is reached
from every thread that initialises or runs an operator: a C++ program drives it from eight threads
under the thread sanitizer (CPU only)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_table_is_safe_with_several_threads(tmp_path):
    exe = tmp_path / "once_per_device"
    built = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread", "-I", str(ROOT / "include"), "-I",
                            str(ROOT / "shflbw_sparse_nn_b200" / "csrc"), str(ROOT / "tests" / "cpp" / "once_per_device_test.cc"),
                            "-o", str(exe), "-pthread"], capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    if "unexpected memory mapping" in run.stderr:
        pytest.skip("the thread sanitizer cannot run on this kernel")
    assert run.returncode == 0 and run.stdout == "ok\n", run.stdout + run.stderr
