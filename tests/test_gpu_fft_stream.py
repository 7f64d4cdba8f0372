"""The streaming FFT pass (16-byte aligned columns, enough tiles to share
twiddles) against the per-tile passes, which columns one word off alignment
take, and against the oracle: every shape it is instantiated with, plain and
low-degree extensions, column counts that leave blocks a ragged last tile.
Which kernel a pass takes is asked of the library, so a change of the rule
that would leave a case to the per-tile kernel fails here (and, for the whole
list, in test_fft_splits.py, without a GPU)."""
import numpy as np
import pytest

import pyoracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
P = (1 << 31) - 1


@pytest.fixture(scope="module")
def B():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gpustark.backend import GpuBackend
    yield GpuBackend
    GpuBackend.fft_reset_tuning()


def columns(g, n, log, off):
    """n columns of 2^log words, `off` words past a 16-byte boundary."""
    stride = (1 << log) + 4
    buf = torch.randint(0, P, (n * stride + 4,), dtype=torch.int32, device="cuda", generator=g)
    return [buf[k * stride + off:k * stride + off + (1 << log)] for k in range(n)]


def host(t):
    return t.cpu().numpy().view(np.uint32)


def edges(cols):
    for k, edge in enumerate((0, P - 1)):
        cols[k % len(cols)][:64] = edge


# (layers, extension, columns, tile log, coalesced bits): contiguous passes of
# 5..13 layers, strided ones of 5 (10/5), 6 (11/5), 7 (12/5), 8 (12/4) and 9
# (13/4) layers, three-pass splits, coefficients shorter than a tile
SHAPES = [(12, 0, 3333, 13, 4), (13, 0, 1601, 13, 4), (13, 1, 801, 13, 4), (12, 1, 1501, 13, 4), (11, 2, 1501, 13, 4),
          (10, 2, 3001, 13, 4), (9, 3, 3003, 13, 4), (8, 4, 3001, 13, 4), (7, 5, 3001, 13, 4), (6, 6, 3001, 13, 4),
          (5, 7, 3001, 13, 4), (14, 0, 777, 12, 4), (16, 1, 95, 13, 4), (18, 0, 49, 13, 4), (18, 2, 13, 13, 4),
          (18, 1, 25, 12, 4), (18, 0, 47, 12, 5), (18, 1, 25, 11, 5), (18, 0, 47, 10, 5), (20, 1, 7, 13, 4),
          (20, 0, 1, 12, 4), (21, 0, 5, 13, 4), (22, 1, 3, 13, 4), (23, 0, 3, 13, 4), (24, 0, 1, 12, 5)]
# Interpolations whose contiguous pass streams: more tiles, since a block of
# one buffer is smaller and more of them are resident (3553 tiles of 2^12
# words, 1777 of 2^13). (layers, columns, tile log, coalesced bits, layers of
# the passes)
INVERSE = [(12, 3601, 13, 4, [12]), (13, 1801, 13, 4, [13]), (12, 3557, 11, 5, [6, 6]), (14, 901, 12, 5, [7, 7]),
           (15, 451, 9, 4, [5, 5, 5]), (16, 227, 12, 4, [8, 8]), (18, 57, 13, 4, [9, 9]), (18, 57, 12, 4, [10, 8]),
           (18, 57, 12, 5, [11, 7]), (20, 15, 12, 4, [12, 8])]


@pytest.mark.parametrize("log,ext,n_cols,tile,coalesce", SHAPES)
def test_stream_passes_equal_tile_passes(B, log, ext, n_cols, tile, coalesce):
    g = torch.Generator(device="cuda")
    g.manual_seed(log * 100 + ext)
    tw = B.precompute_twiddles(max(log + ext, 12) - 1)
    B.fft_set_tuning(0, tile, coalesce)
    assert any(kernel == "stream" for _, _, kernel in B.fft_passes(log + ext, log, n_cols))
    src = columns(g, n_cols, log, 0)
    edges(src)
    off = columns(g, n_cols, log, 1)
    for a, b in zip(off, src):
        a.copy_(b)
    got = B.evaluate_polynomials(src, log + ext, tw, out=columns(g, n_cols, log + ext, 0))
    want = B.evaluate_polynomials(off, log + ext, tw, out=columns(g, n_cols, log + ext, 1))
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert all(torch.equal(a, b) for a, b in zip(src, off))
    if log + ext <= 18:
        for k in {0, n_cols - 1}:
            assert np.array_equal(host(got[k]), O.evaluate(host(src[k]), log + ext))
    B.interpolate_columns(src, log, tw)
    B.interpolate_columns(off, log, tw)
    assert all(torch.equal(a, b) for a, b in zip(src, off))
    # out of place, through the work-list entry's per-size path
    if n_cols <= 3 and log > 13:
        again = columns(g, n_cols, log, 0)
        B.fft_worklist([("interpolate", e, a) for e, a in zip(got, again)], tw) if ext == 0 else None
        if ext == 0:
            B.interpolate_columns(got, log, tw)
            assert all(torch.equal(a, b) for a, b in zip(again, got))


@pytest.mark.parametrize("log,n_cols,tile,coalesce,layers", INVERSE)
def test_stream_interpolations(B, log, n_cols, tile, coalesce, layers):
    g = torch.Generator(device="cuda")
    g.manual_seed(log * 100 + tile)
    tw = B.precompute_twiddles(log - 1)
    B.fft_set_tuning(0, tile, coalesce)
    passes = B.fft_passes(log, n_columns=n_cols, inverse=True)
    assert [p[1] for p in passes] == layers and passes[0][2] == passes[-1][2] == "stream"
    evals = columns(g, n_cols, log, 0)
    edges(evals)
    off = columns(g, n_cols, log, 1)
    for a, b in zip(off, evals):
        a.copy_(b)
    first = {k: host(evals[k]) for k in (0, 1, n_cols - 1)}
    B.interpolate_columns(evals, log, tw)
    B.interpolate_columns(off, log, tw)
    assert all(torch.equal(a, b) for a, b in zip(evals, off))
    for k, values in first.items():
        assert np.array_equal(host(evals[k]), O.interpolate(values, log))
