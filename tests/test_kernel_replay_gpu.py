"""A kernel-level pass in a graph of the caller's, replayed between the state's
own passes: its queue words are its own, so forces and steps afterwards equal a
fresh context's, bit for bit for the FP32 kernels and to 1e-15 of the largest
value for the FP64 atomics (as in the tests of the state's passes).  40,007
bodies: more one-sided items than CTAs, and block pairs enough for the pair
kernel itself, so every kind pulls its items from a queue; 9,000: the forms
without one.  The same for live calls between state passes of every kind.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["accel", "phi"])
@pytest.mark.parametrize("kind", ["pair", "one-sided", "fp64"])
@pytest.mark.parametrize("n", [9000, 40007])
def test_replayed_kernel_call(libkhrr, n, kind, call):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    from khrr.galaxy import make_galaxy
    pos, vel, mass, eps = make_galaxy(n // 3, n - n // 3, 3, eps_dm=0.004).arrays()
    p, m = (torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in (pos, mass))
    e, out = torch.full_like(m, 1e-4), torch.zeros_like(p if call == "accel" else m)
    torch.cuda.synchronize()
    fp64 = khrr.FP64 if kind == "fp64" else 0

    def state_passes(ctx, between):
        """Forces, two steps, forces, one more step, with `between` before each
        pass but the first -> what was downloaded after each."""
        if kind == "pair":
            ctx.set_tuning(128, 8, 128, 0, 2)
        ctx.upload(pos, vel, mass, eps * eps)
        ctx.forces(khrr.ACC | khrr.PHI | fp64)
        got = []
        for run in (lambda: ctx.step(0.002, 2, khrr.PHI | fp64), lambda: ctx.forces(khrr.ACC | khrr.PHI | fp64),
                    lambda: ctx.step(0.002, 1, fp64)):
            between()
            run()
            got.append(ctx.download())
        return got

    with khrr.Context(0) as fresh:
        want = state_passes(fresh, lambda: None)
    with khrr.Context(0) as ctx:
        def kernel_call():
            getattr(ctx, call)(out.data_ptr(), p.data_ptr(), p.data_ptr(), m.data_ptr(), e.data_ptr(), n, khrr.OVERWRITE)

        kernel_call()  # the plan and the buffers, before the capture
        ctx.synchronize()
        first = out.clone()
        stream = torch.cuda.ExternalStream(ctx.stream)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
            kernel_call()

        def replay():
            out.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                g.replay()

        got = state_passes(ctx, replay)
        ctx.synchronize()
        assert torch.equal(out, first) and bool(first.abs().max() > 0)
        for a, b in zip(got, want):
            for k in b:
                assert np.abs(b[k]).max() > 0.0
                assert np.abs(a[k] - b[k]).max() <= (1e-15 if kind == "fp64" else 0.0) * np.abs(b[k]).max(), k
        del g


def test_kinds_and_kernel_calls_in_any_order(libkhrr):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    from khrr.galaxy import make_galaxy
    n = 40007
    pos, vel, mass, eps = make_galaxy(n // 3, n - n // 3, 3, eps_dm=0.006).arrays()
    p, m = (torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in (pos, mass))
    e, out = torch.full_like(m, 1e-4), torch.zeros_like(p)
    torch.cuda.synchronize()

    def run(ctx, kind):
        ctx.set_tuning(128, 8, 128, 0, 2) if kind == "pair" else ctx.set_tuning()
        flags = khrr.FP64 if kind == "fp64" else 0
        ctx.upload(pos, vel, mass, eps * eps)
        ctx.forces(khrr.ACC | khrr.PHI | flags)
        ctx.step(0.002, 2, flags | khrr.PHI)
        return ctx.download()

    want = {}
    for kind in ("pair", "one-sided", "fp64"):
        with khrr.Context(0) as fresh:
            want[kind] = run(fresh, kind)
    with khrr.Context(0) as ctx:
        # the kernel-level call takes the form that the state pass before it set
        for kind in ("pair", "accel", "one-sided", "accel", "fp64", "pair", "fp64", "accel", "pair", "phi", "one-sided"):
            if kind in ("accel", "phi"):
                getattr(ctx, kind)(out.data_ptr(), p.data_ptr(), p.data_ptr(), m.data_ptr(), e.data_ptr(), n, khrr.OVERWRITE)
                continue
            got = run(ctx, kind)
            for k in got:
                a, b = got[k], want[kind][k]
                assert np.abs(a - b).max() <= (1e-15 if kind == "fp64" else 0.0) * np.abs(b).max(), (kind, k)
