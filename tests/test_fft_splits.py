"""FFT pass splits and the kernels of their passes, as the library reports
them without a GPU: the split by size, installed ones (13/4 among them), the
way back, and that the cases of test_gpu_fft_stream.py reach every shape of
the streaming kernel."""
import pytest

pytest.importorskip("torch")

import test_gpu_fft_stream as stream  # noqa: E402
from gpustark.backend import GpuBackend as B  # noqa: E402


@pytest.fixture(autouse=True)
def by_size():
    B.fft_reset_tuning()
    yield
    B.fft_reset_tuning()


def layers(log, coeff_log=None, inverse=False):
    return [p[1] for p in B.fft_passes(log, coeff_log, 1, inverse)]


def test_an_installed_split_is_the_one_that_runs():
    assert layers(18) == [8, 10] and layers(18, inverse=True) == [10, 8]  # by size: 12/4
    assert B.fft_get_tuning(18) == (13, 4)  # nothing installed
    B.fft_set_tuning(18, 13, 4)
    assert layers(18) == [9, 9] and layers(20, 18) == [9, 9] and B.fft_get_tuning(18) == (13, 4)
    assert layers(17) == [7, 10] and layers(19) == [7, 12]  # other sizes go by size
    B.fft_set_tuning(18, 11, 5, extension=2)
    assert layers(20, 18) == [6, 6, 6] and layers(18) == [9, 9]
    B.fft_reset_tuning()
    assert layers(18) == [8, 10] and layers(20, 18) == [8, 10]
    for tile, coalesce in ((13, 4), (12, 4), (12, 5), (10, 5), (6, 0)):
        B.fft_set_tuning(0, tile, coalesce)
        for log in range(3, 29):
            parts = B.fft_passes(log, inverse=True)
            assert [p[0] for p in parts] == [sum(p[1] for p in parts[:k]) for k in range(len(parts))]
            assert sum(p[1] for p in parts) == log and parts[0][1] <= tile
            assert all(p[1] <= tile - coalesce for p in parts[1:]) and len(parts) <= 8


def test_passes_are_refused_outside_the_range():
    from gpustark import GpuStarkError
    for bad in ((0, 0, 1, False), (31, 31, 1, False), (10, 11, 1, False), (10, 9, 1, True), (10, 10, 0, False),
                (10, 10, 65536, False), (10, 0, 1, False)):
        with pytest.raises(GpuStarkError):
            B.fft_passes(*bad)
    assert B.fft_passes(1) == [] and B.fft_passes(2, 1) == []  # closed forms


def test_the_stream_cases_reach_every_shape():
    want = {(lo, n) for lo, sizes in ((False, range(5, 14)), (True, range(5, 10))) for n in sizes}
    seen = {False: set(), True: set()}
    for log, ext, n_cols, tile, coalesce in stream.SHAPES:
        B.fft_set_tuning(0, tile, coalesce)
        seen[False] |= {(lo > 0, n) for lo, n, k in B.fft_passes(log + ext, log, n_cols) if k == "stream"}
    for log, n_cols, tile, coalesce, sizes in stream.INVERSE:
        B.fft_set_tuning(0, tile, coalesce)
        passes = B.fft_passes(log, log, n_cols, True)
        assert [p[1] for p in passes] == sizes and passes[0][2] == passes[-1][2] == "stream"
        seen[True] |= {(lo > 0, n) for lo, n, k in B.fft_passes(log, log, n_cols, True) if k == "stream"}
    assert seen[False] == want and seen[True] == want
