"""Small results that come back through a context's page-locked words: two
contexts in two threads, each with its own state, keep their own sums (the
bits of a single call, whose order of summation is fixed), and a wait that
gave up is reported once, not by the conservation sums after it."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 3072, 200001])
def test_words_of_two_contexts(libkhrr, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    rng = np.random.default_rng(n)
    with khrr.Context(0) as a, khrr.Context(0) as b:
        want, got = [], [[], []]
        for c in (a, b):
            c.upload(rng.standard_normal((n, 3)), rng.standard_normal((n, 3)), rng.random(n) + 0.5, np.full(n, 1e-4))
            want.append(c.conservation())
        assert want[0] != want[1]
        assert khrr.STATUS[a.probe_bounded_wait(0.02)] == "KHRR_ERR_TIMEOUT"

        def calls(k, c):
            for _ in range(20):
                got[k].append(c.conservation())
                c.synchronize()

        threads = [threading.Thread(target=calls, args=(k, c)) for k, c in enumerate((a, b))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k in range(2):
            assert got[k] == [want[k]] * 20
