"""Host arguments on their way into the C ABI, without a GPU: the whole-list
conversions take, wrap and refuse the values that one conversion per value
does."""
import fractions

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from gpustark import _lib as L  # noqa: E402
from gpustark import backend  # noqa: E402


def one_by_one(values):
    arr = (L.QM31 * len(values))(*[backend.qm31(v) for v in values])
    return np.frombuffer(arr, np.uint32).reshape(-1, 4)


ROWS = [[[0, 1, 2**31 - 2, 2**31 - 1]], [[-1, 2**32, 2**32 + 5, -2**31]], [[2**63, 2**64 + 3, -1, 7]],
        [(1, 2, 3, 4), [5, 6, 7, 8]], [[True, False, True, False]], [[1, 2]], [[]], [[1.5, 2.9, -3.5, 4.0]],
        [[2.0**40, 1e19, -1e19, 1.0]], [["1", "22", "3", "4"]], [[fractions.Fraction(7, 2), 2, 3, 4]],
        [[float("nan"), 1, 2, 3]], [[float("inf"), 1, 2, 3]], [[1j, 1, 2, 3]], [[None, 1, 2, 3]], [[1, 2, 3, 4, 5]],
        [["a", 1, 2, 3]], [[1, 2, 3, 4], [1, 2, 3, 4, 5]], [5], [None]]
ROWS += [[np.array(r, dt)] for dt in ("u1", "i2", "u4", "i8", "u8", "f4", "f8", "O") for r in ([1, 2, 3, 4], [9, 8])]
ROWS += [[np.array([2**64 - 1, 2**63, 5, 6], "u8")], [np.array([1e19, 2.0**33, -2.0, 0.5])],
         [np.array([np.nan, 1, 2, 3])], [np.array([1, np.inf, 2, 3])], [np.array([1 + 2j, 1, 2, 3])],
         [[np.float64("nan"), 1, 2, 3]], [[np.float32("inf"), 1, 2, 3]], [[np.complex64(1), 1, 2, 3]], ["1234"],
         [[np.int32(-7), np.uint64(2**64 - 9), np.bool_(True), 3]], [[1, 2], [3, 4, 5, 6, 7, 8]], [np.zeros((2, 2), int)],
         [np.array([-1, -2, 2**62, 3])], [np.arange(4), [2**64, 1, 2, 3]], [np.arange(5)],
         [torch.tensor([1, 2, 3, -4], dtype=torch.int32)], [torch.tensor([1.5, 2.5, 3.5, 4.5], requires_grad=True)]]


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("k", range(len(ROWS)))
def test_qm31_array_equals_one_conversion_per_value(k):
    values = ROWS[k]
    for vals in (values, [[1, 2, 3, 4]] + list(values)):
        try:
            want = one_by_one(vals)
        except Exception as e:
            with pytest.raises(type(e)):
                backend.qm31_array(vals)
            continue
        _, got = backend.qm31_array(vals, len(vals) + 2)
        got = np.frombuffer(got, np.uint32).reshape(-1, 4)
        assert got.shape == (len(vals) + 2, 4) and not got[len(vals):].any()
        assert np.array_equal(got[:len(vals)], want)


class _Library:
    """Stands for the C library: keeps what a call was given."""

    def __init__(self, name, types):
        self.args = None

        def call(*args):
            self.args = [t(a) if t else a for t, a in zip(types, args)]
            return 0

        setattr(self, name, call)


class _Context:
    handle = None


def _host_tensors(monkeypatch):
    empty = torch.empty
    monkeypatch.setattr(backend.torch, "empty", lambda *a, device=None, **k: empty(*a, **k))


def test_worklist_sizes_reach_the_library_as_they_are(monkeypatch):
    """A tensor of no words has no log size; the library refuses it (2^32 - 1)."""
    _host_tensors(monkeypatch)
    some, none = torch.zeros(8, dtype=torch.int32), torch.zeros(0, dtype=torch.int32)
    tw = backend.TwiddleTree(3, some, some)
    lib = _Library("gs_fft_worklist", [None, lambda a: np.ctypeslib.as_array(
        backend.C.cast(a, backend.C.POINTER(backend.C.c_uint32)), (16,)).copy()])
    monkeypatch.setattr(L, "lib", lambda: lib)
    backend.GpuBackend.fft_worklist([("interpolate", some, none), ("evaluate", none, some)], tw, ctx=_Context())
    assert list(lib.args[1][4:7]) == [2**32 - 1, 3, 1] and list(lib.args[1][12:15]) == [3, 2**32 - 1, 0]
    lib = _Library("gs_merkle_worklist", [None, lambda a: np.ctypeslib.as_array(
        backend.C.cast(a, backend.C.POINTER(backend.C.c_uint32)), (12,)).copy()])
    layers = backend.GpuBackend.merkle_worklist([[some, some], [none]], ctx=_Context())
    assert list(lib.args[1][2:4]) == [2, 3] and list(lib.args[1][8:10]) == [1, 2**32 - 1]
    assert [len(x) for x in layers] == [4, 0]


def test_column_indices_wrap_as_a_ctypes_word(monkeypatch):
    _host_tensors(monkeypatch)
    indices = [0, -1, 2**32 + 1, 2**63, -2**70 + 5, np.int64(3)]
    lib = _Library("gs_accumulate_numerators", [None] * 4 + [lambda a: [a[k] for k in range(len(indices))]])
    monkeypatch.setattr(L, "lib", lambda: lib)
    cols = [torch.zeros(8, dtype=torch.int32)]
    backend.GpuBackend.accumulate_numerators(cols, 3, indices, [[0] * 4] * 6, [[0] * 4] * 6, ctx=_Context())
    assert lib.args[4] == [backend.C.c_uint32(int(i)).value for i in indices]
