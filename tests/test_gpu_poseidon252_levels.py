"""Poseidon252 node levels around the sizes where their kernel changes (three
warps per 32 nodes up to a size, a thread per node above it): each level
against the permutation kernel for every node and against the oracle for the
nodes at both ends, children at the edges of the field among them; and whole
proofs over trees whose levels below 32 nodes take one launch."""
import numpy as np
import pytest

import poseidon252 as PS
import pyoracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
EDGES = [0, 1, PS.P - 1, PS.P - 2, (1 << 251) - 1, 1 << 192, (1 << 192) - 1, (PS.P - 1) // 2]


@pytest.fixture(scope="module")
def B():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gpustark.backend import GpuBackend
    return GpuBackend


@pytest.mark.parametrize("log_size", [0, 1, 3, 4, 5, 6, 7, 11, 12, 13, 14])
def test_node_level(B, log_size):
    rng = np.random.default_rng(log_size)
    n = 1 << log_size
    raw = rng.integers(0, 256, (2 * n, 32), dtype=np.uint8)
    raw[:, 0] &= 7  # below the modulus
    for i, v in enumerate(EDGES[:2 * n]):
        raw[-1 - i] = np.frombuffer(PS.to_bytes_be(v), np.uint8)
    out = B.poseidon252_commit_on_layer(log_size, torch.tensor(raw.reshape(-1), device="cuda"), [])
    two = np.frombuffer(PS.to_bytes_be(2), np.uint8)
    states = np.concatenate([raw.reshape(n, 64), np.broadcast_to(two, (n, 32))], axis=1)
    every = B.poseidon252_permute(torch.tensor(states.reshape(-1), device="cuda")).view(n, 3, 32)[:, 0]
    assert torch.equal(out.view(n, 32), every)
    got = out.cpu().numpy().reshape(n, 32)
    for i in sorted({*range(min(n, 5)), *range(max(0, n - 5), n)}):
        children = [int.from_bytes(raw[2 * i + k].tobytes(), "big") for k in range(2)]
        assert got[i].tobytes() == PS.to_bytes_be(PS.permute(children + [2])[0]), i


@pytest.mark.parametrize("log_n", [3, 4, 5, 6])
def test_small_trees(B, log_n):
    from gpustark import prove
    got = prove.prove_wide_fibonacci(log_n, 9, seed=log_n, input_mode=1, merkle_channel="poseidon252")
    assert got == O.prove("wide_fibonacci", log_n, n_cols=9, seed=log_n, input_mode=1,
                         merkle_channel="poseidon252")
