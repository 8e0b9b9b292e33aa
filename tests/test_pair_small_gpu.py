"""The small-layout form of the pair kernel gives the pair kernel's numbers:
every FP32 partial sum has the same terms in the same order, so accelerations
and potentials are equal bit for bit with the pair kernel itself (chunk split
1: the same block pairs, one CTA each), in every form (uniform, per-component
and per-body softenings; one mass per block, short blocks, ragged ends with
ghosts, per-body masses; single and several systems; either output alone) and
on both sides of the line between the two, through the state API and the
kernel-level calls."""
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


def bodies(sizes, eps_d, own_mass):
    from khrr.galaxy import make_galaxy
    parts = [make_galaxy(a, b, 21 + k, eps_dm=eps_d).arrays() for k, (a, b) in enumerate(sizes)]
    pos, vel, mass, eps = (np.concatenate([p[q] for p in parts]) for q in range(4))
    if own_mass:
        mass = mass * np.random.default_rng(1).uniform(0.5, 1.5, mass.size)
    return pos, vel, mass, eps * eps, np.cumsum([0] + [len(p[2]) for p in parts])


@pytest.mark.parametrize("sizes", [[(1, 0)], [(100, 27)], [(128, 896)], [(500, 525)], [(1024, 2048)], [(1536, 4608)],
                                   [(3000, 5003)], [(4096, 8192)], [(4608, 9728)],
                                   [(640, 1408), (100, 30), (1024, 1024), (700, 1501)]])
@pytest.mark.parametrize("eps_d,own_mass", [(0.004, False), (0.007, False), (0.004, True), (0.007, True)])
def test_equal_to_the_pair_kernel(ctx, sizes, eps_d, own_mass):
    import khrr
    pos, vel, mass, eps2, off = bodies(sizes, eps_d, own_mass)
    out = {}
    for split in (0, 1):
        ctx.set_tuning(128, 8, 128, split, 2)
        ctx.upload(pos, vel, mass, eps2, offsets=off)
        for flags in (khrr.ACC, khrr.PHI, khrr.ACC | khrr.PHI):
            ctx.forces(flags)
            out[split, flags] = ctx.download(pos=False, vel=False)
    ctx.set_tuning()
    for flags in (khrr.ACC, khrr.PHI, khrr.ACC | khrr.PHI):
        assert np.array_equal(out[0, flags]["acc"], out[1, flags]["acc"]), flags
        assert np.array_equal(out[0, flags]["phi"], out[1, flags]["phi"]), flags


@pytest.mark.parametrize("n_s,n_d", [(1024, 2048), (1000, 2001), (4096, 8192)])
def test_kernel_level_calls(ctx, n_s, n_d):
    import torch
    import khrr
    pos, _, mass, eps2, _ = bodies([(n_s, n_d)], 0.006, False)
    n = len(mass)
    P, M, E = (torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in (pos, mass, eps2))
    out = {}
    for split in (0, 1):
        ctx.set_tuning(128, 8, 128, split, 2)
        acc, phi = torch.zeros_like(P), torch.zeros_like(M)
        torch.cuda.synchronize()
        ctx.accel(acc.data_ptr(), P.data_ptr(), P.data_ptr(), M.data_ptr(), E.data_ptr(), n, 0)
        ctx.phi(phi.data_ptr(), P.data_ptr(), P.data_ptr(), M.data_ptr(), E.data_ptr(), n, 0)
        ctx.synchronize()
        out[split] = acc.cpu().numpy(), phi.cpu().numpy()
    ctx.set_tuning()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert np.abs(out[0][0]).max() > 0
