"""The tapered pair plan of the FP64 pass, checked on the CPU: every ordered
pair of 128-body tiles of a system exactly once, whatever the sizes
(tests/pair_tiles_check.cpp replays the items of plan_pair_tiles)."""
import os
import subprocess

import pytest

from conftest import PKG, ROOT

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def checker(libkhrr, tmp_path_factory):
    exe = tmp_path_factory.mktemp("plan") / "pair_tiles_check"
    build = PKG / "build"
    cmd = ["g++", "-std=c++20", "-O2", "-I", str(ROOT / "include"), "-I", str(PKG / "csrc"),
           "-I", f"{CUDA}/include", str(ROOT / "tests" / "pair_tiles_check.cpp"), "-o", str(exe),
           "-L", str(build), "-lkhrr", f"-Wl,-rpath,{build}", "-L", f"{CUDA}/lib64", "-lcudart",
           f"-Wl,-rpath,{CUDA}/lib64"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("ctas,sizes", [
    (296, [1]), (296, [127]), (296, [128]), (296, [129]), (296, [1024]), (296, [1025]), (296, [3072]), (296, [10007]),
    (296, [49152]), (296, [131072]), (1, [9000]), (5, [90001]), (296, [1, 1024, 128, 129, 5000, 77, 20480]),
    (296, [4096, 121856, 11264, 1024 * 37 + 512])])
def test_every_tile_pair_once(checker, ctas, sizes):
    r = subprocess.run([str(checker), str(ctas)] + [str(n) for n in sizes], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
    if sizes == [3072]:
        assert r.stdout.split()[2] == "1"  # fewer tiles than the grid's CTAs: one tile per item
