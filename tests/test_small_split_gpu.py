"""The one-sided kernel's split of small systems (one tile per chunk up to a
few): sizes around the 128-body tile, the 512-body i tile and the line where
the split of larger systems takes over, against the FP64 direct sum on the
GPU.  Bound: 2e-6 relative RMS, the small systems' bound of the force tests
(FP32 rounding of the positions), for every shape's dispatch."""
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


@pytest.mark.parametrize("shape", [(128, 4, 1), (256, 2, 1), (128, 8, 0)])
@pytest.mark.parametrize("n", [3, 129, 511, 1025, 8191, 12289, 14336])
def test_forces_of_small_systems(ctx, n, shape):
    import khrr
    from khrr.galaxy import make_galaxy
    pos, vel, mass, eps = make_galaxy(n // 3, n - n // 3, 7, eps_dm=0.006).arrays()
    ctx.set_tuning(shape[0], shape[1], 128, 0, shape[2])
    try:
        ctx.upload(pos, vel, mass, eps * eps)
        ctx.forces(khrr.ACC | khrr.PHI)
        out = ctx.download()
        acc, phi = ctx.accel_fp64_sample(np.arange(n))
    finally:
        ctx.set_tuning()
    assert np.sqrt(((out["acc"] - acc) ** 2).sum() / (acc ** 2).sum()) <= 2e-6
    assert np.sqrt(((out["phi"] - phi) ** 2).sum() / (phi ** 2).sum()) <= 2e-6
