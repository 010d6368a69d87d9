"""Native packing of padded batches against pack_residues of the cut rows: every integer type, ragged and empty rows,
values outside 0..20 in the padding only and within the lengths."""
import numpy as np
import pytest

from pairhmm import _lib


@pytest.fixture(scope='module', autouse=True)
def lib():
    try:
        return _lib.load()
    except _lib.PairHMMError:
        pytest.skip('library not built')


@pytest.mark.parametrize('dtype', ['u1', 'i1', 'u2', 'i2', 'u4', 'i4', 'u8', 'i8'])
def test_equals_cut_rows(dtype):
    rng = np.random.default_rng(3)
    P, wx, wy = 7, 13, 9
    x, y = rng.integers(0, 21, (P, wx)).astype(dtype), rng.integers(0, 21, (P, wy)).astype(dtype)
    Lx, Ly = np.array([0, 13, 1, 5, 0, 12, 7]), np.array([9, 0, 1, 3, 0, 8, 2])
    for p in range(P):   # padding is not looked at
        x[p, Lx[p]:], y[p, Ly[p]:] = 99, 99
    got = _lib.pack_padded(x, y, Lx, Ly)
    want = _lib.pack_residues([v[:n] for v, n in zip(x, Lx)], [v[:n] for v, n in zip(y, Ly)])
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and np.array_equal(a, b)


def test_refusals_and_other_forms():
    x = np.zeros((2, 4), np.int64)
    bad = x.copy()
    bad[1, 2] = 21
    with pytest.raises(ValueError):
        _lib.pack_padded(bad, x, np.array([4, 3]), np.array([1, 1]))
    assert _lib.pack_padded(bad, x, np.array([4, 2]), np.array([1, 1])) is not None
    bad[1, 2] = -1
    with pytest.raises(ValueError):
        _lib.pack_padded(bad, x, np.array([4, 3]), np.array([1, 1]))
    for args in [(x[:, ::2], x, [1, 1], [1, 1]), (x.astype(float), x, [1, 1], [1, 1]), (x, x, [5, 1], [1, 1]),
                 (x, x, [-1, 1], [1, 1]), (list(x), x, [1, 1], [1, 1]), (x, x, [1.0, 1.0], [1, 1]), (x[:0], x[:0], [], [])]:
        assert _lib.pack_padded(args[0], args[1], np.array(args[2]), np.array(args[3])) is None
    empty = _lib.pack_padded(x, x, np.array([0, 0]), np.array([0, 0]))
    assert empty[0].size == 16
