"""One-sided passes over a few thousand bodies: items cut finer than eight
tiles leave one partial per tile, and the reader forms the sums of the
eight-tile chunks from them.  The results are those of the plan that has these
chunks as its items (the split forced), bit for bit, for one mass per tile and
for a mass per body, on the state API and on the caller's device arrays.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 129, 1000, 1024, 2176, 3072, 4097, 7001, 10240, 12000])
@pytest.mark.parametrize("eps_dm", [0.004, 0.008])
def test_same_bits_as_whole_chunks(libkhrr, n, eps_dm):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    from khrr.galaxy import make_galaxy
    ns = n // 3 // 512 * 512 if n % 1024 == 0 else n // 3
    pos, vel, mass, eps = make_galaxy(ns, n - ns, 7, eps_dm=eps_dm).arrays()
    chunks = max(1, (n + 127) // 128 // 8)
    p, m, e = (torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in (pos, mass, eps * eps))
    runs = []
    for split in (0, chunks):
        acc, phi = torch.full_like(p, 0.5), torch.full_like(m, 0.25)
        with khrr.Context(0) as ctx:
            ctx.set_tuning(128, 4, 128, split, 1)
            ctx.upload(pos, vel, mass, eps * eps)
            ctx.forces(khrr.ACC | khrr.PHI)
            out = [ctx.download()[k] for k in ("acc", "phi")]
            ctx.step(0.002, 3, khrr.PHI)
            out += [ctx.download()[k] for k in ("pos", "vel", "acc", "phi")]
            torch.cuda.synchronize()
            for flags in (khrr.OVERWRITE, 0):
                ctx.accel(acc.data_ptr(), p.data_ptr(), p.data_ptr(), m.data_ptr(), e.data_ptr(), n, flags)
                ctx.phi(phi.data_ptr(), p.data_ptr(), p.data_ptr(), m.data_ptr(), e.data_ptr(), n, flags)
                ctx.synchronize()
                out += [acc.cpu().numpy(), phi.cpu().numpy()]
        runs.append(out)
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
