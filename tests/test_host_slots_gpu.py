"""The page-locked words of more contexts than one page has slots for, in use at
the same time, and again after some were closed: each context reads its own
sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_many_contexts(libkhrr):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr

    def make(k):
        c = khrr.Context(0)
        c.upload(np.eye(3), np.full((3, 3), k + 1.0), np.ones(3), np.full(3, 1e-4))
        return c

    held = {k: make(k) for k in range(18)}
    for round_ in range(2):
        for k, c in held.items():
            assert c.conservation()["Ix"] == 3.0 * (k + 1)
            c.synchronize()
        for k in (0, 5, 16):
            held[k].close()
            held[k] = make(k)
    for c in held.values():
        c.close()
