"""khrr_forces in a capture of the caller's: the reset of the queue and of the
accumulated sums is part of the graph, so its replays do not depend on what the
context ran in between, and a capture that never ran leaves the context's own
passes right.  FP32 results bit for bit, FP64 atomics to 1e-15 of the largest.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["pair", "one-sided", "fp64"])
def test_captured_forces(libkhrr, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    from khrr.galaxy import make_galaxy
    n = 9000
    flags = khrr.ACC | khrr.PHI | (khrr.FP64 if kind == "fp64" else 0)
    first, second = (make_galaxy(3000, n - 3000, seed, eps_dm=0.004).arrays() for seed in (3, 4))
    p, m = (torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in (first[0], first[2]))
    e, out = torch.full_like(m, 1e-4), torch.zeros_like(p)
    with khrr.Context(0) as ctx:
        if kind == "pair":
            ctx.set_tuning(128, 8, 128, 0, 2)

        def state(bodies, run):
            ctx.upload(bodies[0], bodies[1], bodies[2], bodies[3] ** 2)
            run()
            ctx.synchronize()
            got = ctx.download()
            return got["acc"], got["phi"]

        def same(a, b):
            for x, y in zip(a, b):
                assert np.abs(x - y).max() <= (1e-15 if kind == "fp64" else 0.0) * np.abs(y).max()

        def other():  # a kernel-level pass leaves the shared queue as it ended
            torch.cuda.synchronize()
            ctx.accel(out.data_ptr(), p.data_ptr(), p.data_ptr(), m.data_ptr(), e.data_ptr(), n, khrr.OVERWRITE)

        want = [state(b, lambda: ctx.forces(flags)) for b in (first, second)]
        assert np.abs(want[0][0]).max() > 0.0 and not np.array_equal(want[0][0], want[1][0])
        stream = torch.cuda.ExternalStream(ctx.stream)
        g = torch.cuda.CUDAGraph()
        other()
        with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
            ctx.forces(flags)
        same(state(first, lambda: ctx.forces(flags)), want[0])

        def replay():
            other()
            with torch.cuda.stream(stream):
                g.replay()
                g.replay()

        same(state(second, replay), want[1])
        same(state(first, lambda: ctx.forces(flags)), want[0])
        del g
