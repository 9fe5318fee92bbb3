"""Growth of the library's prefill scratch (csrc/grow.h), against an allocator that refuses what is too large."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_grow_buffer(tmp_path):
    exe = str(tmp_path / "grow_buffer")
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "p100e_engine_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cabi", "grow_buffer.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
