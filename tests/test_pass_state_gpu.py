"""State carried between calls: the force kernels' queue and sums, zeroed by
the kernel that reads them, and the conservation kernel's block counter.

  * passes of different kinds in any order on one context (pair, one-sided,
    plain, FP64 in both forms, kernel-level calls, timed steps) give what a
    fresh context gives: bit for bit for the FP32 kernels, whose results are
    reproducible, to 1e-15 of the largest value for the FP64 atomics;
  * the conservation sums at block edges and beyond one block per SM slot,
    against float64 numpy to 1e-12 of the sum of absolute terms, twice the
    same bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def khrr_mod(libkhrr):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    return khrr


def bodies(n, seed=5):
    from khrr.galaxy import make_galaxy
    pos, vel, mass, eps = make_galaxy(n // 3, n - n // 3, seed, eps_dm=0.006).arrays()
    return pos, vel, mass, eps * eps


def run_kind(khrr, ctx, kind, data):
    """One set-up pass and two steps of a kind -> downloaded state."""
    ctx.set_tuning(128, 8, 128, 0, 2) if kind.startswith("pair") else ctx.set_tuning()
    flags = {"fp64": khrr.FP64, "plain": khrr.PLAIN}.get(kind, 0)
    ctx.enable_timing(kind.endswith("timed"))
    ctx.upload(*data)
    ctx.forces(khrr.ACC | khrr.PHI | flags)
    ctx.step(0.002, 2, flags | khrr.PHI)
    ctx.step(0.002, 1, flags)
    ctx.enable_timing(False)
    return ctx.download()


def test_passes_in_any_order(khrr_mod):
    import torch
    data = bodies(2500)
    order = ["pair", "one-sided", "fp64", "pair timed", "plain", "fp64", "accel", "one-sided", "pair", "accel", "pair"]
    with khrr_mod.Context(0) as ctx:
        for kind in order:
            if kind == "accel":
                p, m, e = (torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in (data[0], data[2], data[3]))
                out = torch.zeros_like(p)
                torch.cuda.synchronize()
                ctx.accel(out.data_ptr(), p.data_ptr(), p.data_ptr(), m.data_ptr(), e.data_ptr(), len(data[2]), 16)
                ctx.synchronize()
                continue
            got = run_kind(khrr_mod, ctx, kind, data)
            with khrr_mod.Context(0) as fresh:
                want = run_kind(khrr_mod, fresh, kind.split()[0], data)
            for k in want:
                if kind == "fp64":
                    assert np.abs(got[k] - want[k]).max() <= 1e-15 * np.abs(want[k]).max(), (kind, k)
                else:
                    assert np.array_equal(got[k], want[k]), (kind, k)


@pytest.mark.parametrize("n", [1, 255, 257, 4096, 151552, 160001])
def test_conservation_at_block_edges(khrr_mod, n):
    rng = np.random.default_rng(n)
    pos, vel = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    mass = rng.uniform(0.5, 1.5, n)
    with khrr_mod.Context(0) as ctx:
        ctx.upload(pos, vel, mass, np.full(n, 1e-4))
        a, b = ctx.conservation(), ctx.conservation()
    assert a == b
    c = np.cross(pos, vel) * mass[:, None]
    for k, terms in (("Lx", c[:, 0]), ("Ly", c[:, 1]), ("Lz", c[:, 2]), ("Ix", mass * vel[:, 0]),
                     ("Ek", mass * (vel * vel).sum(1))):
        assert abs(a[k] - terms.sum()) <= 1e-12 * np.abs(terms).sum(), k
    assert a["Ep"] == 0.0 and a["E"] == 0.5 * a["Ek"]
    r = np.hypot(pos[:, 0], pos[:, 1])
    assert abs(a["R_max"] - r.max()) <= 1e-15 * r.max()
    assert a["Z_max"] == np.abs(pos[:, 2]).max() and a["Vz_max"] == np.abs(vel[:, 2]).max()
