"""The host threads of the whole-lattice transfers, without a GPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_two_transfers_at_once(tmp_path):
    exe = str(tmp_path / "copy_pool")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I" + os.path.join(CUDA, "include"), "-x", "c++",
                    os.path.join(ROOT, "tests", "cxx", "copy_pool.cpp"), "-o", exe,
                    "-L" + os.path.join(CUDA, "lib64"), "-lcudart", "-Wl,-rpath," + os.path.join(CUDA, "lib64")],
                   check=True, timeout=300)
    # two jobs that overwrite each other copy a part of one only, or wait for good
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
