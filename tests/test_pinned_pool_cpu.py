"""What the pool of pinned host memory keeps: bounded, by the largest allowance of a
device (picard_gpu_pool_keep names one), and given back with the last context."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pinned_pool(tmp_path):
    exe = str(tmp_path / "pinned_pool")
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "-pthread", "-I",
                    os.path.join(ROOT, "picard_b200", "csrc"), os.path.join(ROOT, "tests", "pinned_pool.cpp"), "-o",
                    exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout
