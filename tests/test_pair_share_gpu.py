"""The pair kernel's share per SM: whatever number of items an SM is given
(one, fewer than one per SM, a few, many; items of unequal time from short
blocks and own-block tiles), every item runs exactly once.  The sums are
fixed-point and do not depend on who runs an item, so against the FP64 direct
sum a lost or repeated item of k bodies shows as an error of order k / n;
bound 2e-6 relative RMS, the small systems' bound of the force tests."""
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


@pytest.mark.parametrize("sizes", [[(300, 700)], [(4096, 12288)], [(12000, 8003)], [(1536, 2560), (640, 1408), (512, 15360)],
                                   [(512, 1024)] * 40])
def test_every_item_runs_once(ctx, sizes):
    import khrr
    from khrr.galaxy import make_galaxy
    parts = [make_galaxy(a, b, 11 + k, eps_dm=0.006).arrays() for k, (a, b) in enumerate(sizes)]
    pos, vel, mass, eps = (np.concatenate([p[q] for p in parts]) for q in range(4))
    ctx.upload(pos, vel, mass, eps * eps, offsets=np.cumsum([0] + [len(p[2]) for p in parts]))
    want, phi = ctx.accel_fp64_sample(np.arange(len(mass)))
    for _ in range(2):  # the second pass starts from what the first left
        ctx.forces(khrr.ACC | khrr.PHI)
        out = ctx.download()
        assert np.sqrt(((out["acc"] - want) ** 2).sum() / (want ** 2).sum()) <= 2e-6
        assert np.sqrt(((out["phi"] - phi) ** 2).sum() / (phi ** 2).sum()) <= 2e-6
