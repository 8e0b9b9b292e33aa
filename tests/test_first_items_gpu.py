"""One-sided kernel and per-body kernels of small systems: a pass whose items
fit the grid (none comes from the queue) beside ones with more items than
CTAs, and slot counts around the eight that the sums are read by.  Twice on
one context, for the second pass meets what the first left in the queue.
Bound: 2e-6 relative RMS against the FP64 direct sum on the GPU, the small
systems' bound of the force tests; the two passes agree bit for bit, since
the split fixes the order of every sum."""
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
    yield c
    c.close()


@pytest.mark.parametrize("n,split", [(2, 1), (1000, 7), (1024, 8), (2500, 9), (2500, 17), (9000, 64), (37887, 1),
                                     (37889, 8), (40000, 17)])
def test_items_and_slots(ctx, n, split):
    import khrr
    from khrr.galaxy import make_galaxy
    pos, vel, mass, eps = make_galaxy(n // 3, n - n // 3, 11, eps_dm=0.006).arrays()
    ctx.set_tuning(128, 4, 128, split, 1)
    try:
        ctx.upload(pos, vel, mass, eps * eps)
        ctx.forces(khrr.ACC | khrr.PHI)
        first = ctx.download()
        ctx.forces(khrr.ACC | khrr.PHI)
        again = ctx.download()
        some = np.arange(0, n, max(1, n // 2000))
        acc, phi = ctx.accel_fp64_sample(some)
    finally:
        ctx.set_tuning()
    for k in ("acc", "phi"):
        assert np.array_equal(first[k], again[k])
    assert np.sqrt(((first["acc"][some] - acc) ** 2).sum() / (acc ** 2).sum()) <= 2e-6
    assert np.sqrt(((first["phi"][some] - phi) ** 2).sum() / (phi ** 2).sum()) <= 2e-6
