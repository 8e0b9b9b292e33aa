"""Step graphs of a program that changes dt with every call: the memory they take
stays bounded, and the steps are those of contexts that make one step at a time
(bit for bit, one graph kept or many dropped in between)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def host_mb():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * 4096 / 1e6


def test_changing_dt(libkhrr):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    from khrr.galaxy import make_galaxy
    pos, vel, mass, eps = make_galaxy(300, 707, 3, eps_dm=0.006).arrays()
    dts = [1e-4 + 1e-6 * k for k in range(70)]
    dts = [d for k, d in enumerate(dts) for d in (d, dts[0], dts[max(0, k - 40)])]  # new, often and seldom used ones

    def run(parts):
        with khrr.Context(0) as ctx:
            ctx.upload(pos, vel, mass, eps * eps)
            ctx.forces(khrr.ACC)
            for dt in dts:
                for m in parts:
                    ctx.step(dt, m)
            return ctx.download()

    a, b = run([3]), run([1, 1, 1])
    for k in ("pos", "vel", "acc"):
        assert np.array_equal(a[k], b[k]), k

    with khrr.Context(0) as ctx:
        ctx.upload(pos, vel, mass, eps * eps)
        ctx.forces(khrr.ACC)
        marks = []
        for k in range(600):
            ctx.step(1e-6 + 1e-9 * k, 8)
            if k in (199, 599):
                ctx.synchronize()
                marks.append((torch.cuda.mem_get_info()[0] / 1e6, host_mb()))
        # 400 graphs more took about 60 MB of each.
        assert marks[0][0] - marks[1][0] < 20.0 and marks[1][1] - marks[0][1] < 20.0, marks
