"""The page-locked words of contexts across device resets.  On the CPU the pool
itself against a fake allocator (tests/host_words_check.cpp includes
khrr-nbody_b200/csrc/host_words.h); on the GPU a program that resets its device
between contexts, in a process of its own."""
import subprocess
import sys

import pytest

from conftest import PKG, ROOT


def test_pool_against_a_fake(tmp_path):
    exe = tmp_path / "host_words_check"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(PKG / "csrc"),
                        str(ROOT / "tests" / "host_words_check.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


PROGRAM = """
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import numpy as np, khrr
runtime = ctypes.CDLL("libcudart.so.12")
for k in range(3):
    with khrr.Context(0) as a, khrr.Context(0) as b:
        for c, v in ((a, k + 1.0), (b, k + 11.0)):
            c.upload(np.eye(3), np.full((3, 3), v), np.ones(3), np.full(3, 1e-4))
        assert a.conservation()["Ix"] == 3.0 * (k + 1) and b.conservation()["Ix"] == 3.0 * (k + 11)
    assert runtime.cudaDeviceReset() == 0
print("ok")
"""


@pytest.mark.gpu
def test_contexts_between_resets(libkhrr):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(PKG)], capture_output=True, text=True, timeout=120,
                       env={**__import__("os").environ, "LD_LIBRARY_PATH": "/usr/local/cuda/lib64"})
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
