"""accumulate_numerators and batch_eval_at_point around the edges of their
tensor-core kernels: tiles of 512 rows, chunks of 16 columns in operand stages
of 32, groups of 128 polynomials, words equal to P, outputs or columns that the
16-byte accesses cannot take."""
import ctypes as C

import numpy as np
import pytest

from stwo_b200 import B200Backend, DeviceColumn, ffi
from stwo_b200.backend import NumeratorTerm, SampleBatch, _ptr_array, _words

pytestmark = pytest.mark.gpu
P = (1 << 31) - 1


class View:
    def __init__(self, buf, offset, log_size):
        self.buf, self.ptr, self.log_size = buf, buf.ptr + 4 * offset, log_size


def words(rng, n):
    v = rng.integers(0, P, n, dtype=np.uint32)
    v[rng.integers(0, n, max(1, n // 8))] = P
    return v


@pytest.mark.parametrize("log_n", [8, 9, 10, 13])
@pytest.mark.parametrize("n_terms", [1, 2, 3, 7, 8, 9, 16, 17, 31, 33, 48, 255, 257, 258, 259])
def test_numerators_tiles_and_chunks(oracle, log_n, n_terms):
    rng = np.random.default_rng(100 * log_n + n_terms)
    cols = [words(rng, 1 << log_n) for _ in range(min(n_terms, 20))]
    cols[0][:] = P
    terms = [(k % len(cols), rng.integers(0, P, 4, dtype=np.uint32), rng.integers(0, P, 4, dtype=np.uint32))
             for k in range(n_terms)]
    point = rng.integers(0, P, 8, dtype=np.uint32)
    (out, first), = B200Backend().accumulate_numerators([DeviceColumn.from_host(c) for c in cols], [(point, terms)])
    ref, ref_first = oracle.accumulate_numerators(cols, log_n, point, terms)
    assert (first == ref_first).all()
    for a, b in zip(out.to_host(), ref):
        assert (a == b).all()


@pytest.mark.parametrize("in_off,out_off", [(1, 0), (0, 1), (4, 4)])
def test_numerators_alignment(oracle, in_off, out_off):
    rng = np.random.default_rng(7 + in_off)
    log_n, n = 10, 1 << 10
    cols = [words(rng, n) for _ in range(5)]
    dev = [View(DeviceColumn.from_host(np.concatenate([np.zeros(in_off, np.uint32), c])), in_off, log_n) for c in cols]
    outs = [View(DeviceColumn(n + out_off), out_off, log_n) for _ in range(4)]
    point = rng.integers(0, P, 8, dtype=np.uint32)
    terms = [(k, rng.integers(0, P, 4, dtype=np.uint32), rng.integers(0, P, 4, dtype=np.uint32)) for k in range(5)]
    arr, batch, first = (NumeratorTerm * 5)(), (SampleBatch * 1)(), (C.c_uint32 * 4)()
    for k, (i, v, a) in enumerate(terms):
        arr[k].column_index, arr[k].sample_value, arr[k].random_coeff = i, _words(v, 4), _words(a, 4)
    batch[0].point, batch[0].terms, batch[0].n_terms = _words(point, 8), C.cast(arr, C.POINTER(NumeratorTerm)), 5
    ffi.init()
    ffi.call("stwo_b200_accumulate_numerators", _ptr_array(dev), C.c_uint32(5), C.c_uint32(log_n), batch, C.c_uint32(1),
             _ptr_array(outs), first, None)
    ref, _ = oracle.accumulate_numerators(cols, log_n, point, terms)
    for o, r in zip(outs, ref):
        assert (o.buf.to_host()[out_off:] == r).all()


# 2^12 takes the chunked kernel; the tensor cores (whole groups of 128, short
# ones, several buckets a block) and the bucket kernel on both sides of the line
BATCH_EVAL = [(12, n) for n in (1, 31, 32, 33, 127, 128, 129, 300)]
BATCH_EVAL += [(13, n) for n in (1, 31, 32, 33, 127, 128, 129, 300, 1024)]
BATCH_EVAL += [(14, n) for n in (1, 31, 32, 33, 127, 128, 129, 300, 600, 1024)]
BATCH_EVAL += [(15, 300), (16, 148), (16, 149), (16, 256), (16, 257)]
BATCH_EVAL += [(17, n) for n in (1, 31, 32, 33, 74, 75, 76, 127, 128, 129, 149, 300)]
BATCH_EVAL += [(18, 74), (18, 76), (18, 128), (18, 129), (19, 96), (19, 260)]


@pytest.mark.parametrize("log_n,n_polys", BATCH_EVAL)
def test_batch_eval_groups(oracle, log_n, n_polys):
    rng = np.random.default_rng(1000 * log_n + n_polys)
    polys = [words(rng, 1 << log_n) for _ in range(min(n_polys, 9))]
    polys[0][:] = P
    dev = [DeviceColumn.from_host(p) for p in polys]
    point = rng.integers(1, P, 8, dtype=np.uint32)
    got = B200Backend().batch_eval_at_point([dev[k % len(dev)] for k in range(n_polys)], point)
    want = [B200Backend().eval_at_point(d, point) for d in dev]  # the integer-pipe kernels
    for k in range(n_polys):
        assert (got[k] == want[k % len(dev)]).all(), k
    assert (want[1 % len(dev)] == oracle.eval_at_secure_point(polys[1 % len(dev)], point)).all()
