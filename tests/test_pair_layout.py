"""The one-pair path's device block, without a GPU: a small program asks the
library for the block's layout over sizes around the ones where the walk's
records move to global memory, and checks that every part has room for what the
kernels write to it."""
import os
import subprocess

from tweakseq_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_parts_have_room(tmp_path):
    B.build()
    exe = str(tmp_path / "pair_layout_check")
    r = subprocess.run([B.nvcc(), "-std=c++17", "-I", os.path.join(B.ROOT, "include"), "-I", B.CSRC,
                        os.path.join(HERE, "cpp", "pair_layout_check.cpp"), "-o", exe, "-L", B.LIBDIR, "-ltsq_gb300",
                        "-Xlinker", "-rpath=" + B.LIBDIR], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "layout ok", r.stdout[:2000]
