"""The cloud-in-cell deposit and gather, two lanes per body, where the deposit
spreads over extra meshes and where it does not: meshes from 2^3 (every body
near a face) on, body counts at warp and block edges and on both sides of the
rule's lines, bodies outside the mesh, repeated deposits into the same cells
(they accumulate, and leave the extra meshes zero) and a captured deposit.
Deposits against the oracle to 1e-12 of the largest cell (FP64 sums in another
order), gathers bit for bit."""
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


@pytest.mark.parametrize("n,nx", [(1, 2), (15, 3), (16, 2), (129, 5), (1000, 8), (4097, 16), (20001, 32), (60000, 33),
                                  (3000, 40)])
def test_deposit_and_gather(ctx, oracle, n, nx):
    import torch
    import khrr
    rng = np.random.default_rng(n)
    L, cs = 2.0, 4.0 / nx
    pos = rng.normal(scale=0.7, size=(n, 3))
    pos[:: max(1, n // 7)] *= 4.0  # some outside
    mass = rng.uniform(0.5, 1.5, n)
    P, M = torch.as_tensor(pos, device="cuda"), torch.as_tensor(mass, device="cuda")
    cells = torch.zeros(nx ** 3, dtype=torch.float64, device="cuda")
    mesh = khrr.Mesh.make((-L,) * 3, (cs,) * 3, (nx,) * 3)
    torch.cuda.synchronize()
    want = oracle.cic_deposit(pos, mass, (-L,) * 3, (cs,) * 3, (nx,) * 3)
    for k in (1, 2, 3):  # the extra meshes come in with the second deposit
        ctx.cic_deposit(P.data_ptr(), M.data_ptr(), n, mesh, cells.data_ptr())
        ctx.synchronize()
        assert np.abs(cells.cpu().numpy() - k * want).max() <= 1e-12 * k * np.abs(want).max()
    cacc, cval = rng.normal(size=(nx ** 3, 3)), rng.normal(size=nx ** 3)
    A, V = torch.as_tensor(cacc, device="cuda"), torch.as_tensor(cval, device="cuda")
    out_a, out_v = torch.full((n, 3), 7.0, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.cic_gather(P.data_ptr(), n, mesh, A.data_ptr(), V.data_ptr(), out_a.data_ptr(), out_v.data_ptr())
    ctx.synchronize()
    wa, wv = oracle.cic_gather(pos, (-L,) * 3, (cs,) * 3, (nx,) * 3, cacc, cval)
    assert np.array_equal(out_a.cpu().numpy(), wa) and np.array_equal(out_v.cpu().numpy(), wv)
    out_v.zero_()
    torch.cuda.synchronize()
    ctx.cic_gather(P.data_ptr(), n, mesh, None, V.data_ptr(), None, out_v.data_ptr())
    ctx.synchronize()
    assert np.array_equal(out_v.cpu().numpy(), wv)


def test_captured_deposit(ctx, oracle):
    """Inside the caller's capture the deposit keeps no pointer of the context's."""
    import torch
    import khrr
    rng = np.random.default_rng(3)
    n, nx = 30000, 32
    pos, mass = rng.normal(scale=0.5, size=(n, 3)), rng.uniform(0.5, 1.5, n)
    P, M = torch.as_tensor(pos, device="cuda"), torch.as_tensor(mass, device="cuda")
    cells = torch.zeros(nx ** 3, dtype=torch.float64, device="cuda")
    mesh = khrr.Mesh.make((-2.0,) * 3, (4.0 / nx,) * 3, (nx,) * 3)
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx.set_stream(s.cuda_stream)
    try:
        with torch.cuda.graph(g, stream=s):
            ctx.cic_deposit(P.data_ptr(), M.data_ptr(), n, mesh, cells.data_ptr())
        g.replay()
        g.replay()
        torch.cuda.synchronize()
    finally:
        ctx.set_stream(None)
    want = 2 * oracle.cic_deposit(pos, mass, (-2.0,) * 3, (4.0 / nx,) * 3, (nx,) * 3)
    assert np.abs(cells.cpu().numpy() - want).max() <= 1e-12 * np.abs(want).max()
