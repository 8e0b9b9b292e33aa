"""The symmetric FP64 pass over its tile classes and operand ranges against
the one-sided FP64 pass (rsqrt() and per-body masses throughout): tiles of
one mass and softening, a component border inside a tile, a ragged end,
masses or softenings of each body's own, and coordinates and softenings
inside and outside the range of the r^-3 series.  Both are FP64 sums of the
same terms in another order: the terms agree to ~4 ulp and 10^4 of them are
summed, so 1e-13 of the largest term bounds the difference."""
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


@pytest.mark.parametrize("n_s,n_d,eps_d,own,scale", [
    (1024, 2048, 0.004, "", 1.0),       # whole blocks, one softening
    (1536, 2560, 0.008, "", 1.0),       # a block of two classes
    (1500, 2501, 0.008, "", 1.0),       # a tile of two classes, a ragged end
    (1024, 2048, 0.004, "mass", 1.0),
    (1024, 2048, 0.004, "eps", 1.0),
    (1500, 2500, 0.008, "", 1e80),      # inside the series' range
    (1500, 2500, 0.008, "", 1e100),     # coordinates beyond it
    (1500, 2500, 0.008, "", 1e-90),     # softenings below it
    (1024, 2048, 0.004, "one far", 1.0)])
def test_symmetric_pass_equals_the_one_sided_one(ctx, monkeypatch, n_s, n_d, eps_d, own, scale):
    import khrr
    from khrr.galaxy import make_galaxy
    pos, vel, mass, eps = make_galaxy(n_s, n_d, 91, eps_dm=eps_d).arrays()
    pos, eps2 = pos * scale, (eps * scale) ** 2
    rng = np.random.default_rng(91)
    if own == "mass":
        mass = mass * rng.uniform(0.5, 1.5, mass.size)
    if own == "eps":
        eps2 = eps2 * rng.uniform(0.5, 1.5, mass.size)
    if own == "one far":
        pos[2000] = (3e90, -1e90, 0.0)
    out = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("KHRR_FP64_ONESIDED", mode)
        ctx.upload(pos, vel, mass, eps2)
        ctx.forces(khrr.ACC | khrr.PHI | khrr.FP64)
        out[mode] = ctx.download()
        ctx.forces(khrr.ACC | khrr.FP64)
        out[mode]["acc only"] = ctx.download()["acc"]
    for k in ("acc", "phi", "acc only"):
        a, b = out["0"][k], out["1"][k]
        assert np.isfinite(b).all()
        assert np.abs(a - b).max() <= 1e-13 * np.abs(b).max(), k
