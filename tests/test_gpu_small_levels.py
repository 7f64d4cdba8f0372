"""Tree levels, FRI layers and channel steps of at most 32 hashes, which take
four lanes per compression, and the hand-over from the wider levels: every
level of trees around the kernels' unit sizes, and whole proofs whose FRI
layers start at each size of the single-launch tail."""
import hashlib

import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def G():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gpustark import prove
    return prove


@pytest.mark.parametrize("top", [1, 2, 4, 5, 6, 7, 8, 9, 10, 11, 14, 15, 16, 18])
def test_every_level_of_a_tree(G, top):
    from gpustark.backend import GpuBackend as B
    g = torch.Generator(device="cuda")
    g.manual_seed(top)
    layers = [torch.empty(8 << k, dtype=torch.int32, device="cuda") for k in range(top)]
    leaves = torch.randint(-2**31, 2**31 - 1, (8 << top,), dtype=torch.int32, device="cuda", generator=g)
    B.commit_node_layers(layers + [leaves])
    below = leaves.cpu().numpy().tobytes()
    for k in reversed(range(top)):
        got = layers[k].cpu().numpy().tobytes()
        want = b"".join(hashlib.blake2s(below[64 * i:64 * i + 64]).digest() for i in range(1 << k))
        assert got == want, k
        below = got


@pytest.mark.parametrize("log_n", [3, 4, 5, 6, 7, 8, 9, 10, 11])
@pytest.mark.parametrize("last", [0, 2])
def test_tails_of_every_size(G, log_n, last):
    cfg = G.pcs_config(pow_bits=2, log_blowup=1, n_queries=5, log_last_layer=last)
    got = G.prove_wide_fibonacci(log_n, 5, seed=log_n, config=cfg)
    assert got == O.prove("wide_fibonacci", log_n, n_cols=5, seed=log_n, pow_bits=2, n_queries=5, log_blowup=1,
                          log_last_layer=last)
