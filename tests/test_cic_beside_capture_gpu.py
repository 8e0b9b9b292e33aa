"""Deposits on the context's stream while the thread captures another stream, in
the capture mode that forbids allocations: the deposits run, the extra meshes'
allocation with the second of them included, and the capture is as it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_deposits_beside_a_capture(libkhrr, oracle):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    rng = np.random.default_rng(5)
    n, nx = 30000, 32
    pos, mass = rng.normal(scale=0.5, size=(n, 3)), rng.uniform(0.5, 1.5, n)
    P, M = torch.as_tensor(pos, device="cuda"), torch.as_tensor(mass, device="cuda")
    cells = torch.zeros(nx ** 3, dtype=torch.float64, device="cuda")
    mesh = khrr.Mesh.make((-2.0,) * 3, (4.0 / nx,) * 3, (nx,) * 3)
    x = torch.ones(1000, device="cuda")
    g = torch.cuda.CUDAGraph()
    with khrr.Context(0) as ctx:
        ctx.cic_deposit(P.data_ptr(), M.data_ptr(), n, mesh, cells.data_ptr())  # loads the kernels
        torch.cuda.synchronize()
        with torch.cuda.graph(g, capture_error_mode="global"):
            x.mul_(2.0)
            for _ in range(3):
                ctx.cic_deposit(P.data_ptr(), M.data_ptr(), n, mesh, cells.data_ptr())
            x.add_(1.0)
        ctx.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert bool((x == 3.0).all())
        want = 4 * oracle.cic_deposit(pos, mass, (-2.0,) * 3, (4.0 / nx,) * 3, (nx,) * 3)
        assert np.abs(cells.cpu().numpy() - want).max() <= 1e-12 * want.max()
