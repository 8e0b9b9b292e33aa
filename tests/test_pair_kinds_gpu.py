"""Pair kernels where a tile's bodies share mass and softening, one of them, or
neither: every form has the general form's terms, so results do not depend on
which one ran.

One body q sits so far away (1e18) that its force on the others is exactly
zero and its potential lost in rounding.  With a softening larger than the
others' it makes its tile, and the warp that holds it, take the general form
without changing any term that counts: the other bodies keep their bits.
Against the FP64 direct sum on the GPU the bound is 2e-6 relative RMS, the
small systems' bound of the force tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(libkhrr):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    c = khrr.Context(0)
    c.set_tuning(128, 8, 128, 0, 2)
    yield c
    c.close()


@pytest.mark.parametrize("n", [1025, 5003, 15001, 24576])
@pytest.mark.parametrize("kinds", ["one", "two masses", "two softenings"])
@pytest.mark.parametrize("q", [0, 127, 128, 1024 + 517, -1])
def test_forms_agree(ctx, n, kinds, q):
    import khrr
    from khrr.galaxy import make_galaxy
    q = min(q, n - 2) if q >= 0 else n - 1
    pos, vel, _, _ = make_galaxy(n // 3, n - n // 3, 7).arrays()
    first = np.arange(n) < n // 3
    mass = np.full(n, 1.0 / n)
    eps2 = np.full(n, 1.6e-5)
    if kinds == "two masses":
        mass[first] *= 3.0
    if kinds == "two softenings":
        eps2[first] *= 2.0
    pos = pos.copy()
    pos[q] = (1e18, 0.0, 0.0)
    outs = []
    for e in (eps2[q], 6.4e-5):
        e2 = eps2.copy()
        e2[q] = e
        ctx.upload(pos, vel, mass, e2)
        for flags in (khrr.ACC, khrr.ACC | khrr.PHI):
            ctx.forces(flags)
            outs.append(ctx.download())
    rest = np.arange(n) != q
    assert np.array_equal(outs[0]["acc"][rest], outs[2]["acc"][rest])
    assert np.array_equal(outs[1]["acc"][rest], outs[3]["acc"][rest])
    assert np.array_equal(outs[1]["phi"][rest], outs[3]["phi"][rest])
    some = np.flatnonzero(rest)[:: max(1, n // 1000)]
    acc, phi = ctx.accel_fp64_sample(some)
    assert np.sqrt(((outs[3]["acc"][some] - acc) ** 2).sum() / (acc ** 2).sum()) <= 2e-6
    assert np.sqrt(((outs[3]["phi"][some] - phi) ** 2).sum() / (phi ** 2).sum()) <= 2e-6
