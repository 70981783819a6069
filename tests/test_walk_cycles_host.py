"""A walk's end by a cycle, on the CPU: walk_to_end of the device code,
compiled for the host, against the plain loop of iterations over made-up walks
(tests/c/walk_cycles.cpp)."""
import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_walk_to_end_equals_the_plain_loop(tmp_path):
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    exe = tmp_path / "walk_cycles"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-w", f"-I{cuda}",
                    f"-I{ROOT / 'include'}", f"-I{ROOT / 'voxelg_b200' / 'csrc'}",
                    str(ROOT / "tests" / "c" / "walk_cycles.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
