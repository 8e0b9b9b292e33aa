"""The cloud-in-cell gather for each choice of outputs (accelerations and value,
either alone, neither), whose kernels differ in the lanes per body: body counts
at warp and block edges, bodies outside the mesh; bit for bit against the
oracle, and an output that is not asked for stays as it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nx", [(1, 2), (15, 3), (129, 5), (4097, 16), (30001, 33)])
def test_outputs(libkhrr, oracle, n, nx):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    rng = np.random.default_rng(n)
    L, cs = 2.0, 4.0 / nx
    pos = rng.normal(scale=0.7, size=(n, 3))
    pos[:: max(1, n // 7)] *= 4.0
    cacc, cval = rng.normal(size=(nx ** 3, 3)), rng.normal(size=nx ** 3)
    wa, wv = oracle.cic_gather(pos, (-L,) * 3, (cs,) * 3, (nx,) * 3, cacc, cval)
    P, A, V = (torch.as_tensor(x, device="cuda") for x in (pos, cacc, cval))
    mesh = khrr.Mesh.make((-L,) * 3, (cs,) * 3, (nx,) * 3)
    with khrr.Context(0) as ctx:
        for acc, val in ((True, True), (True, False), (False, True), (False, False)):
            a = torch.full((n, 3), 7.0, dtype=torch.float64, device="cuda")
            v = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            ctx.cic_gather(P.data_ptr(), n, mesh, A.data_ptr(), V.data_ptr(), a.data_ptr() if acc else None,
                           v.data_ptr() if val else None)
            ctx.synchronize()
            assert np.array_equal(a.cpu().numpy(), wa if acc else np.full((n, 3), 7.0)), (acc, val)
            assert np.array_equal(v.cpu().numpy(), wv if val else np.full(n, 7.0)), (acc, val)
