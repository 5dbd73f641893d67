"""The kernels' shared-memory limits under threads (csrc/lmb_smem.h), on the
host: tests/cpp/smem_limit_selftest.cpp."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
BINARY = os.path.join(HERE, "cpp", "_build", "smem_limit_selftest")


def test_limit_is_never_lowered_between_threads():
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "cpp"), BINARY], check=True)
    out = subprocess.run([BINARY], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
