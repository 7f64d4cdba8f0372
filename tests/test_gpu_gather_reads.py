"""Gathers that store into mapped host memory, with few indices by value: the
counts around both rules (16 indices, 1 MiB), repeated and boundary indices,
and reads that follow the kernel that writes the data without a wait."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def B():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gpustark.backend import GpuBackend
    return GpuBackend


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 300, 32768, 32769])
def test_hashes(B, n):
    rng = np.random.default_rng(n)
    for log in (0, 5, 12):
        layer = torch.randint(-2**31, 2**31 - 1, (8 << log,), dtype=torch.int32, device="cuda")
        idx = rng.integers(0, 1 << log, n).astype(np.uint32)
        idx[-1], idx[0] = 0, (1 << log) - 1
        layer.add_(1)  # enqueued just before the read
        got = B.batch_get_hashes(layer, idx)
        want = layer.view(-1, 8)[torch.from_numpy(idx.astype(np.int64)).cuda()].cpu().numpy()
        assert np.array_equal(got, want.view(np.uint8).reshape(-1, 32))


@pytest.mark.parametrize("n_cols,n", [(1, 1), (3, 16), (7, 17), (64, 4096), (64, 4097)])
def test_values(B, n_cols, n):
    rng = np.random.default_rng(n)
    cols = [torch.randint(0, 2**31 - 1, (1 << 13,), dtype=torch.int32, device="cuda") for _ in range(n_cols)]
    idx = rng.integers(0, 1 << 13, n).astype(np.uint32)
    got = np.asarray(B.batch_at_multi(cols, idx)).view(np.uint32).reshape(n, n_cols)
    at = torch.from_numpy(idx.astype(np.int64)).cuda()
    want = torch.stack([c[at] for c in cols], dim=1).cpu().numpy().view(np.uint32)
    assert np.array_equal(got, want)
