"""The pair kernel's tile list on the host: the rules of mfree_kernels.cuh are
compiled into a small program (tests/tile_list_host.cu) and checked there, over
the levels at which each of them cuts a tile."""
import os
import subprocess

from iwf_mfree_gpu_3d_b200 import build

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "tile_list_host.cu")


def test_tile_list_rules(tmp_path):
    exe = str(tmp_path / "tile_list_host")
    r = subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-I" + build.INCLUDE, "-I" + build.CSRC, SRC, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
