"""The host side of the calls: the words of numerator terms, and buffers that
are parts of one allocation."""
import ctypes as C

import numpy as np
import pytest

from stwo_b200 import backend as B


@pytest.mark.parametrize("form", [lambda w: np.array(w, np.uint32), lambda w: w, tuple,
                                  lambda w: np.array(w, np.int64), lambda w: np.array(w, np.uint32).reshape(2, 2),
                                  lambda w: np.array([[x, 7] for x in w], np.uint32)[:, 0]])
def test_terms_are_the_structures(form):
    words = np.random.default_rng(3).integers(0, 1 << 31, (5, 9)).tolist()
    terms = [(np.int64(w[0]), form(w[1:5]), form(w[5:])) for w in words]
    arr = B._terms(terms)
    got = C.cast(C.c_void_p(arr.ctypes.data), C.POINTER(B.NumeratorTerm))
    for k, w in enumerate(words):
        assert [got[k].column_index, *got[k].sample_value, *got[k].random_coeff] == w


def test_terms_refused():
    v = np.zeros(4, np.uint32)
    assert B._terms([]).shape == (1, 9)
    assert B._terms([(-1, v, v)])[0, 0] == 0xFFFFFFFF  # out of range for the library, which says so
    for bad in ([(0, v)], [(0, v, v, v)], [(0, v, v), (0, v)]):
        with pytest.raises(ValueError):
            B._terms(bad)
    for bad in ([(0, v[:3], v)], [(0, v, [1, 2, 3, 4, 5])]):
        with pytest.raises(AssertionError):
            B._terms(bad)


@pytest.mark.gpu
@pytest.mark.parametrize("log", [0, 3, 17, 18, 19])
def test_parts_of_a_buffer(log):
    n = 1 << log
    bufs = B.SecureColumn.empty(n).cols + B._tree_layers(min(log, 17), None)
    sizes = [4 * n] * 4 + [32 << k for k in range(min(log, 17) + 1)]
    assert [b.nbytes for b in bufs] == sizes
    for k, b in enumerate(bufs):
        assert b.ptr % 256 == 0
        b.upload(np.full(b.nbytes, k + 1, np.uint8))
    bufs[0].close()
    bufs[0].close()
    del bufs[4]
    for k, b in zip([2, 3, 4, *range(6, len(sizes) + 1)], bufs[1:]):
        assert (b.download(np.uint8) == k).all()
