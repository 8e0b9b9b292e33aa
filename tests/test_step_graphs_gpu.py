"""Steps share a graph up to eight at a time: any number of steps in one call
gives the bits of as many calls of one step (the FP32 kernels' sums are
reproducible), with the potential of the last step alone, timed or not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(128, 4, 1), (128, 8, 2)])
@pytest.mark.parametrize("nsteps", [2, 7, 8, 9, 17])
def test_steps_of_one_call(libkhrr, nsteps, shape):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    from khrr.galaxy import make_galaxy
    pos, vel, mass, eps = make_galaxy(500, 1003, 3, eps_dm=0.006).arrays()
    outs = []
    for parts, timed in (([nsteps], False), ([1] * nsteps, False), ([nsteps], True), ([3, nsteps - 3], False)):
        if min(parts) < 1:
            continue
        with khrr.Context(0) as ctx:
            ctx.set_tuning(shape[0], shape[1], 128, 0, shape[2])
            ctx.enable_timing(timed)
            ctx.upload(pos, vel, mass, eps * eps)
            ctx.forces(khrr.ACC | khrr.PHI)
            # the passes that carry the potential fold their sums otherwise
            for k, m in enumerate(parts):
                ctx.step(0.002, m, khrr.PHI if k == len(parts) - 1 else 0)
            outs.append(ctx.download())
    for o in outs[1:]:
        for k in ("pos", "vel", "acc", "phi"):
            assert np.array_equal(outs[0][k], o[k]), k
