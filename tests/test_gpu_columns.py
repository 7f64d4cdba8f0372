"""Column lists of every spacing: evenly spaced ones (in either direction, with
gaps, one column, the same column repeated) reach the kernels as a base and a
stride, all others through a pointer table; both give the oracle's results."""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# rows of a matrix, as the columns of a call
PICKS = {"rows": [0, 1, 2, 3, 4], "reversed": [7, 6, 5, 4], "gaps": [1, 4, 7], "one": [3], "pair": [5, 2],
         "uneven": [0, 1, 3, 4], "zigzag": [0, 2, 1, 3, 2], "repeated": [6, 6, 6], "nearly": [0, 1, 2, 3, 4, 5, 7]}


@pytest.fixture(scope="module")
def B():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gpustark.backend import GpuBackend
    return GpuBackend


def host(t):
    return t.detach().cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("pick", PICKS)
@pytest.mark.parametrize("log,off", [(3, 0), (6, 0), (6, 3), (13, 0)])
def test_column_spacings(B, pick, log, off):
    rng = np.random.default_rng(log * 10 + off)
    n, idx = 1 << log, PICKS[pick]
    words = rng.integers(0, O.P, (8, n + 4), dtype=np.int64).astype(np.uint32)
    mat = torch.from_numpy(words.view(np.int32)).cuda()
    cols = [mat[i, off:off + n] for i in idx]
    ref = [words[i, off:off + n].copy() for i in idx]
    leaves = B.commit_on_layer(log, None, cols)
    assert np.array_equal(host(leaves).view(np.uint8).reshape(-1, 32), O.commit_on_layer(log, None, ref))
    tw = B.precompute_twiddles(log)
    out = B.evaluate_polynomials(cols, log + 1, tw)  # separate allocations
    want = O.evaluate_columns(ref, log + 1, root_log=log)
    assert all(np.array_equal(host(a), b) for a, b in zip(out, want))
    point = [int(v) for v in rng.integers(0, O.P, 8)]
    assert B.batch_eval_at_point(cols, point) == [list(map(int, O.eval_at_point(c, point))) for c in ref]
    if len(set(idx)) == len(idx):  # in place: distinct columns
        B.interpolate_columns(cols, log, tw)
        want = O.interpolate_columns(ref, log, root_log=log)
        assert all(np.array_equal(host(a), b) for a, b in zip(cols, want))
        rest = [i for i in range(8) if i not in idx]
        assert np.array_equal(host(mat[rest]), words[rest])


@pytest.mark.parametrize("log,n_cols", [(4, 3), (9, 17), (12, 40), (17, 24), (18, 1), (18, 24), (18, 25)])
@pytest.mark.parametrize("off", [0, 1])
def test_layer_kernels(B, log, n_cols, off):
    """A layer over children and columns by either kernel (aligned or not, few
    and more columns, small and large layers), evenly spaced or not."""
    rng = np.random.default_rng(log * 100 + n_cols)
    n = 1 << log
    words = rng.integers(0, O.P, (n_cols, n + 4), dtype=np.int64).astype(np.uint32)
    prev = rng.integers(0, 256, (2 * n, 32), dtype=np.uint8)
    mat = torch.from_numpy(words.view(np.int32)).cuda()
    kids = torch.from_numpy(prev.reshape(-1).view(np.int32)).cuda()
    for order in (list(range(n_cols)), [0] + list(range(n_cols - 1, 0, -1)) + [0]):
        ref = [words[i, off:off + n].copy() for i in order]
        got = B.commit_on_layer(log, kids, [mat[i, off:off + n] for i in order])
        assert np.array_equal(host(got).view(np.uint8).reshape(-1, 32), O.commit_on_layer(log, prev.reshape(-1), ref))
