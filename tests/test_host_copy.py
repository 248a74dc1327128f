"""Host-side copies of the engine (csrc/host_copy.h), compiled on their own: no GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_host_copies(tmp_path):
    exe = str(tmp_path / "host_copy_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", os.path.join(ROOT, "tinyllama.cpp_b200", "csrc"),
                    os.path.join(ROOT, "tests", "abi", "host_copy_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
