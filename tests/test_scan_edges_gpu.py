"""The prefix sums at the edges of their segments (2 or 4 cells), warps (256),
the reference's blocks (512) and tiles (4096), both views, exact against
numpy: {count, start_id} pairs through khrr_compute_prefix_sums, plain counts
through khrr_bin."""
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


@pytest.mark.parametrize("ncells", [1, 2, 3, 63, 255, 257, 511, 513, 1023, 4095, 4096, 4097, 12289, 100003, 4096 * 1025 + 7])
@pytest.mark.parametrize("mode", [0, 1])
def test_pairs(ctx, ncells, mode):
    import torch
    rng = np.random.default_rng(ncells)
    count = rng.integers(0, 9, ncells).astype(np.int32)
    pairs = torch.zeros((ncells + 4, 2), dtype=torch.int32, device="cuda")
    pairs[:, 1] = -7
    pairs[:ncells, 0] = torch.as_tensor(count)
    nb = (ncells + 511) // 512
    pbc = torch.full((nb + 1,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx.compute_prefix_sums(pairs.data_ptr(), pbc.data_ptr(), ncells, mode)
    ctx.synchronize()
    got = pairs.cpu().numpy()
    incl = np.cumsum(count, dtype=np.int64)
    blocks = incl[np.minimum(np.arange(1, nb + 1) * 512, ncells) - 1]
    before = np.concatenate([[0], blocks])[np.arange(ncells) // 512]
    assert np.array_equal(got[:ncells, 0], count)
    assert np.array_equal(got[:ncells, 1], before if mode == 0 else incl - count)
    assert np.array_equal(got[ncells:], [[0, -7]] * 4)
    assert np.array_equal(pbc.cpu().numpy(), np.concatenate([blocks, [-7]]))


@pytest.mark.parametrize("nx", [1, 2, 5, 8, 16, 17, 33])
def test_plain_counts(ctx, nx):
    rng = np.random.default_rng(nx)
    pos = rng.uniform(-1, 1, (3000, 3))
    ctx.upload(pos, np.zeros_like(pos), np.ones(3000), np.full(3000, 1e-4))
    b = ctx.bin((-1.0,) * 3, (2.0 / nx,) * 3, (nx,) * 3)
    incl = np.cumsum(b["count"], dtype=np.int64)
    assert incl[-1] == 3000 and np.array_equal(b["start"], incl - b["count"])
    assert np.array_equal(b["count"], np.bincount(b["cell_id"], minlength=nx ** 3))
