"""The z-marching stencil kernels at the sizes where their packs, rows, blocks
and z ranges end, bit for bit against the oracle's restatements: the FP64
step through khrr_wave_iteration (pairs of cells for even nx and 16-byte
aligned arrays, single cells otherwise: both must give the same bits) and the
FP32 step through khrr_wave_solve (packs of four for nx % 4 == 0)."""
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


@pytest.mark.parametrize("nx", [3, 4, 5, 6, 17, 34, 66, 95, 130])
@pytest.mark.parametrize("shift", [0, 1])
def test_fp64_step(ctx, oracle, nx, shift):
    import torch
    import khrr
    C = nx ** 3
    rng = np.random.default_rng(nx)
    phi, old, mass = rng.normal(size=C), rng.normal(size=C), rng.uniform(0.0, 1e-3, C)
    W, Wo = khrr.WaveParams.make(nx, 8.0 / nx), oracle.wave_params(nx, 8.0 / nx)
    dev = []
    for a in (np.zeros(C), phi, old, mass):
        t = torch.zeros(C + 2, dtype=torch.float64, device="cuda")  # shift 1: 8-byte aligned only
        t[shift:shift + C] = torch.as_tensor(a)
        dev.append(t)
    torch.cuda.synchronize()
    ctx.wave_iteration(*(t.data_ptr() + 8 * shift for t in dev), W)
    ctx.synchronize()
    got = dev[0].cpu().numpy()
    assert np.array_equal(got[shift:shift + C], oracle.wave_iter_f64(Wo, phi, old, mass))
    assert not got[:shift].any() and not got[shift + C:].any()


@pytest.mark.parametrize("nx", [3, 4, 8, 12, 33, 36, 68, 102, 132])
def test_fp32_steps(ctx, oracle, nx):
    import khrr
    rng = np.random.default_rng(nx)
    n = 500
    pos, mass = rng.uniform(-3.9, 3.9, (n, 3)), rng.uniform(0.5, 1.5, n)
    ctx.upload(pos, np.zeros((n, 3)), mass, np.full(n, 1e-4))
    m32 = ctx.bin((-4.0,) * 3, (8.0 / nx,) * 3, (nx,) * 3)["cell_mass"].astype(np.float32)
    it, _, phi = ctx.wave_solve(khrr.WaveParams.make(nx, 8.0 / nx), tol=0.0, max_iter=7, check_every=3, cold=True)
    Wo = oracle.wave_params(nx, 8.0 / nx)
    prev, cur = np.zeros(nx ** 3, np.float32), np.zeros(nx ** 3, np.float32)
    for _ in range(7):
        prev, cur = cur, oracle.wave_iter_f32(Wo, cur, prev, m32)
    assert it == 7 and np.array_equal(phi, cur)
