"""The lines between the pair kernel and its form for few block pairs, with one
mass per block and without: on both sides of each the numbers are the pair
kernel's (chunk split 1: the same block pairs, one CTA each) bit for bit, by
the state API and by the kernel-level calls, whose masses may change between
calls of one size."""
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


# (stars, dark) per system: 14 | 15, 17 to 19 | 20 blocks of one mass; 16, 21 | 22
# blocks of mixed ones; 11 short and long blocks of several systems.
@pytest.mark.parametrize("sizes", [[(4096, 10240)], [(5120, 10240)], [(6144, 11264)], [(7168, 12288)], [(8192, 12288)],
                                   [(5000, 11001)], [(7000, 9930)], [(7000, 14400)], [(7000, 15001)],
                                   [(6000, 9000), (640, 128), (1500, 1501)]])
def test_equal_on_both_sides(ctx, sizes):
    import torch
    import khrr
    from khrr.galaxy import make_galaxy
    parts = [make_galaxy(a, b, 31 + k, eps_dm=0.006).arrays() for k, (a, b) in enumerate(sizes)]
    pos, vel, mass, eps = (np.concatenate([p[q] for p in parts]) for q in range(4))
    eps2, off, n = eps * eps, np.cumsum([0] + [len(p[2]) for p in parts]), len(mass)
    other = mass * np.random.default_rng(2).uniform(0.5, 1.5, n)
    P, E = (torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in (pos, eps2))
    out = {}
    for split in (0, 1):
        ctx.set_tuning(128, 8, 128, split, 2)
        ctx.upload(pos, vel, mass, eps2, offsets=off)
        for flags in (khrr.ACC, khrr.ACC | khrr.PHI):
            ctx.forces(flags)
            out.setdefault(split, []).append(ctx.download(pos=False, vel=False))
        for m in (mass, other, mass):
            M = torch.as_tensor(m, device="cuda")
            acc = torch.zeros_like(P)
            torch.cuda.synchronize()
            ctx.accel(acc.data_ptr(), P.data_ptr(), P.data_ptr(), M.data_ptr(), E.data_ptr(), n, 0)
            ctx.synchronize()
            out[split].append({"acc": acc.cpu().numpy()})
    ctx.set_tuning()
    assert all(np.abs(o["acc"]).max() > 0 for o in out[0])
    for a, b in zip(out[0], out[1]):
        for k in a:
            assert np.array_equal(a[k], b[k])
