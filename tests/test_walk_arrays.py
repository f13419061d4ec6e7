"""CPU tests of how the Python binding hands walk arrays to the C ABI."""
import ctypes

import numpy as np
import pytest
import torch

from research_codes_gb300 import _lib, abi, functors


def _addresses(arrs):
    return [v or 0 for v in functors._ptr_array(arrs)][:len(arrs)]


class _Sub(np.ndarray):
    pass


@pytest.mark.parametrize("make", [
    lambda a: a, tuple,
    lambda a: [x if k % 3 else x[:0] for k, x in enumerate(a)],        # empty ones: null
    lambda a: [x.view(_Sub) if k == 2 else x for k, x in enumerate(a)],
    lambda a: [], lambda a: a[:1],
], ids=["list", "tuple", "empties", "subclass", "none", "one"])
def test_addresses_of_walk_arrays(make):
    arrs = make([np.zeros(3 + k, abi.HydroEPJ) for k in range(40)])
    assert _addresses(arrs) == [a.ctypes.data if len(a) else 0 for a in arrs]


def test_addresses_of_rows_that_exist_for_the_loop_alone():
    """A 2-D array of walks, and a sequence that makes its arrays on access."""
    m = np.zeros((7, 5), abi.GravityEPI)
    assert _addresses(m) == [m.ctypes.data + k * m.strides[0] for k in range(7)]

    class Lazy:
        def __len__(self):
            return 7

        def __getitem__(self, k):
            return m[k]

    assert _addresses(Lazy()) == [m.ctypes.data + k * m.strides[0] for k in range(7)]


def test_counts():
    for c in ([], [3], (1, 2, 3), np.arange(5), np.arange(5, dtype=np.uint8), [2.0, 7.0]):
        assert list(functors._count_array(c))[:len(c)] == [int(x) for x in c]


class _Int:
    def __int__(self):
        return 4


@pytest.mark.parametrize("counts", [
    np.array([np.nan, 1.0]), np.array([np.inf]), [float("nan")], [None], np.array(["2020"], "M8[Y]"),
    np.array([[1], [2]]), {2: 1, 3: 1}, [2 ** 70 + 3, 1], [2 ** 63, -1], np.array([2 ** 63 + 5], np.uint64),
    ["3", b"7"], [True, _Int()], np.array([1.5, 2.0]), torch.tensor([1, 2]), [torch.tensor(3), torch.tensor([4])],
    [np.int64(7), np.int32(-2)], (2 ** 31, 5), [3, np.float64(3.7)], (np.uint64(2 ** 63 + 9),),
], ids=str)
def test_counts_are_taken_as_int_takes_them(counts):
    """What int() refuses is refused, what it accepts is accepted (low 32 bits)."""
    try:
        want = [ctypes.c_int32(int(c)).value for c in counts]
    except (TypeError, ValueError, OverflowError) as e:
        with pytest.raises(type(e)):
            functors._count_array(counts)
    else:
        assert list(functors._count_array(counts)) == want


def test_the_binding_helper_is_not_part_of_the_abi():
    assert "sph_member_pointers" not in _lib.header_functions()
    obj = (ctypes.c_int64 * 4)(1, 2, 3, 4)
    base = ctypes.addressof(obj)
    out = (ctypes.c_void_p * 2)()
    src = (ctypes.c_void_p * 2)(base, base + 16)
    _lib.load().sph_member_pointers(ctypes.cast(src, ctypes.c_void_p), 2, 8, out)
    assert list(out) == [2, 4]
