"""The FP64 step with its planes streamed through shared memory (even nx from 178
to 352, 16-byte aligned arrays), bit for bit: against the oracle at the
smallest size, and against the march of single cells, which 8-byte aligned
arrays take, where segments, rows and z ranges end in all ways; the arrays'
neighbours stay untouched, and phi_new may be phi_old.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def step(ctx, khrr, torch, nx, shift, fields, in_place=False):
    C = nx ** 3
    dev = []
    for a in fields:
        t = torch.full((C + 4,), 7.0, dtype=torch.float64, device="cuda")
        t[shift:shift + C] = a
        dev.append(t)
    torch.cuda.synchronize()
    phi, old, mass = (t.data_ptr() + 8 * shift for t in dev)
    out = dev[1] if in_place else torch.full((C + 4,), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.wave_iteration(out.data_ptr() + 8 * shift, phi, old, mass, khrr.WaveParams.make(nx, 8.0 / nx))
    ctx.synchronize()
    assert (out[:shift] == 7.0).all() and (out[shift + C:] == 7.0).all()
    return out[shift:shift + C]


@pytest.mark.parametrize("nx", [176, 178, 180, 198, 200, 222, 256, 302, 350, 352, 354])
def test_same_bits_as_the_march(libkhrr, nx):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    g = torch.Generator(device="cuda").manual_seed(nx)
    fields = [torch.randn(nx ** 3, dtype=torch.float64, device="cuda", generator=g) for _ in range(2)]
    fields.append(torch.rand(nx ** 3, dtype=torch.float64, device="cuda", generator=g) * 1e-3)
    with khrr.Context(0) as ctx:
        want = step(ctx, khrr, torch, nx, 1, fields)
        assert torch.equal(step(ctx, khrr, torch, nx, 0, fields), want)
        assert torch.equal(step(ctx, khrr, torch, nx, 2, fields), want)
        assert torch.equal(step(ctx, khrr, torch, nx, 0, fields, in_place=True), want)


def test_oracle(libkhrr, oracle):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import khrr
    nx = 178
    rng = np.random.default_rng(1)
    a = [rng.normal(size=nx ** 3), rng.normal(size=nx ** 3), rng.uniform(0.0, 1e-3, nx ** 3)]
    with khrr.Context(0) as ctx:
        got = step(ctx, khrr, torch, nx, 0, [torch.as_tensor(x, device="cuda") for x in a]).cpu().numpy()
    assert np.array_equal(got, oracle.wave_iter_f64(oracle.wave_params(nx, 8.0 / nx), *a))
