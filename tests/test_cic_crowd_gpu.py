"""The cloud-in-cell deposit's choice, on the device, between the mesh and its
extra meshes: bodies spread evenly, with a few pairs in the sample that it goes
by (on both sides of its line), crowded throughout, crowded only in the last
or the first blocks, sums that cancel, in turns on one context (the extra meshes
and the words end as they began); and two contexts that deposit into one mesh at
the same time.  Against the oracle to 1e-12 of the sum of |m w| in the fullest
cell (FP64 sums in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L, NX, N = 2.0, 32, 60001


@pytest.fixture(scope="module")
def khrr_mod(libkhrr):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    return khrr


def bodies(kind, n=N):
    rng = np.random.default_rng(len(kind))
    pos, mass = rng.uniform(-L, L, (n, 3)), rng.uniform(0.5, 1.5, n)
    if kind == "crowded":
        pos = rng.normal(scale=0.1, size=(n, 3))
    elif kind == "crowded at the end":
        pos[-n // 4:] = rng.uniform(0.13, 0.24, (n - n * 3 // 4, 3))
    elif kind == "crowded at the start":
        pos[:300] = rng.uniform(0.13, 0.24, (300, 3))
    elif kind.startswith("pairs"):  # of the sample's 256 bodies, so many pairs share a place
        k, at = int(kind[-1]), np.arange(256) * (n // 256)
        pos[at[1:2 * k:2]] = pos[at[0:2 * k:2]]
    elif kind == "cancelling":
        pos[1::2] = pos[:-1:2] = rng.uniform(0.13, 0.5, (n // 2, 3))
        mass[1::2] = -mass[:-1:2]
    return pos, mass


def mesh_of(khrr, nx=NX):
    return khrr.Mesh.make((-L,) * 3, (2 * L / nx,) * 3, (nx,) * 3)


# 32^3: spread always; 88^3: by the sample (four extra meshes).
@pytest.mark.parametrize("nx,n", [(NX, N), (88, 500003)])
def test_kinds_in_turn(khrr_mod, oracle, nx, n):
    import torch
    kinds = ["pairs %d" % k for k in range(9)] + ["even", "crowded", "even", "crowded at the end", "crowded at the start", "cancelling", "even", "crowded"]
    with khrr_mod.Context(0) as ctx:
        mesh = mesh_of(khrr_mod, nx)
        cells = torch.zeros(nx ** 3, dtype=torch.float64, device="cuda")
        for kind in ["crowded"] + kinds:  # the extra meshes come in with the second deposit
            pos, mass = bodies(kind, n)
            P, M = torch.as_tensor(pos, device="cuda"), torch.as_tensor(mass, device="cuda")
            cells.zero_()
            torch.cuda.synchronize()
            ctx.cic_deposit(P.data_ptr(), M.data_ptr(), len(mass), mesh, cells.data_ptr())
            ctx.synchronize()
            want = oracle.cic_deposit(pos, mass, (-L,) * 3, (2 * L / nx,) * 3, (nx,) * 3)
            scale = oracle.cic_deposit(pos, np.abs(mass), (-L,) * 3, (2 * L / nx,) * 3, (nx,) * 3).max()
            assert np.abs(cells.cpu().numpy() - want).max() <= 1e-12 * scale, kind


def test_two_contexts_one_mesh(khrr_mod, oracle):
    import torch
    parts = [bodies("crowded"), bodies("crowded at the end")]
    want = sum(oracle.cic_deposit(p, m, (-L,) * 3, (2 * L / NX,) * 3, (NX,) * 3) for p, m in parts)
    on = [tuple(torch.as_tensor(x, device="cuda") for x in pm) for pm in parts]
    cells = torch.zeros(NX ** 3, dtype=torch.float64, device="cuda")
    mesh = mesh_of(khrr_mod)
    with khrr_mod.Context(0) as a, khrr_mod.Context(0) as b:
        for _ in range(40):
            cells.zero_()
            torch.cuda.synchronize()
            for _ in range(3):
                for ctx, (p, m) in zip((a, b), on):
                    ctx.cic_deposit(p.data_ptr(), m.data_ptr(), N, mesh, cells.data_ptr())
            a.synchronize()
            b.synchronize()
            assert np.abs(cells.cpu().numpy() - 3 * want).max() <= 1e-12 * 3 * want.max()
