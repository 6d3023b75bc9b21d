"""The bounded device waits of the tensor-core kernels give up cleanly.

The composition, OODS and quotient kernels wait on mbarriers for their blocks'
tensor-core products; every wait polls a bounded number of times.  Here the
bound is set to zero polls, so the first wait of every thread runs out: the
kernel sets the prover's error flag, stores no more rows, waits for the products
still in flight and leaves, and the prove returns STWO_B200_ETIMEOUT with a
message.  Nothing faults, and the same prover then proves the same inputs with
the default bound, byte for byte as the oracle.
"""
import ctypes as C

import numpy as np
import pytest

from stwo_b200 import DeviceColumn, SecureColumn, WideFibProver, ffi, sync, wide_fib_config
from stwo_b200.backend import NumeratorTerm, SampleBatch, _ptr_array, _terms, _words

pytestmark = pytest.mark.gpu
P = (1 << 31) - 1
ETIMEOUT = -4


@pytest.mark.parametrize("log_n,cols", [(12, 100), (16, 24)])
def test_stream_wait_timeout_reports_and_recovers(oracle, log_n, cols):
    a, b = oracle.wide_fib_inputs(log_n, 4242 + log_n)
    ref = oracle.prove_wide_fib(oracle.wide_fib_config(log_n, cols), a, b)
    prover = WideFibProver(wide_fib_config(log_n, cols))
    da, db = DeviceColumn.from_host(a), DeviceColumn.from_host(b)
    assert prover.prove(da, db) == ref
    prover.set_stream_spin(0)
    with pytest.raises(ffi.B200Error) as e:
        prover.prove(da, db)
    assert e.value.code == ETIMEOUT
    assert "column stream" in str(e.value)
    prover.set_stream_spin(WideFibProver.STREAM_SPIN_DEFAULT)
    assert prover.prove(da, db) == ref
    assert prover.prove(da, db) == ref
    prover.close()


# The stand-alone entries: 0 polls, so that every wait of their tensor-core
# forms runs out.  A failure belongs to the call that met it: no later call or
# sync, of its own stream or of another, reports it.

@pytest.mark.parametrize("log_n,n_terms", [(9, 107), (13, 40), (17, 130), (10, 300)])
def test_numerators_without_polls_are_whole(oracle, log_n, n_terms):
    r = np.random.default_rng(log_n)
    cols = [r.integers(0, P + 1, 1 << log_n, dtype=np.uint32) for _ in range(min(n_terms, 20))]
    terms = [(k % len(cols), r.integers(0, P, 4, dtype=np.uint32), r.integers(0, P, 4, dtype=np.uint32))
             for k in range(n_terms)]
    point = r.integers(0, P, 8, dtype=np.uint32)
    dev = [DeviceColumn.from_host(c) for c in cols]
    out = SecureColumn.empty(1 << log_n)
    arr, batch, first = _terms(terms), (SampleBatch * 1)(), (C.c_uint32 * 4)()
    batch[0].point, batch[0].n_terms = _words(point, 8), n_terms
    batch[0].terms = C.cast(C.c_void_p(arr.ctypes.data), C.POINTER(NumeratorTerm))
    ref, ref_first = oracle.accumulate_numerators(cols, log_n, point, terms)
    for polls in (0, WideFibProver.STREAM_SPIN_DEFAULT, 0):
        for c in out.cols:
            c.upload(np.full(1 << log_n, P, np.uint32))
        ffi.call("stwo_b200_accumulate_numerators_polls", _ptr_array(dev), C.c_uint32(len(dev)), C.c_uint32(log_n),
                 batch, C.c_uint32(1), _ptr_array(out.cols), first, C.c_uint32(polls), None)
        sync()
        assert list(first) == list(ref_first)
        for a, b in zip(out.to_host(), ref):
            assert (a == b).all(), polls


def test_batch_eval_timeout_is_its_own_calls(oracle):
    import torch
    r = np.random.default_rng(5)
    log_n, n = 18, 128  # the tensor-core form
    polys = [r.integers(0, P, 1 << log_n, dtype=np.uint32) for _ in range(3)]
    dev = [DeviceColumn.from_host(p) for p in polys]
    point = r.integers(1, P, 8, dtype=np.uint32)
    want = [oracle.eval_at_secure_point(p, point) for p in polys]
    streams = [torch.cuda.Stream() for _ in range(2)]

    def call(stream, polls):
        out = (C.c_uint32 * (4 * n))(*([7] * (4 * n)))
        try:
            ffi.call("stwo_b200_batch_eval_at_point_polls", _ptr_array([dev[k % 3] for k in range(n)]), C.c_uint32(n),
                     C.c_uint32(log_n), _words(point, 8), out, C.c_uint32(polls), C.c_void_p(stream.cuda_stream))
        except ffi.B200Error as e:
            assert list(out) == [7] * (4 * n)
            return e.code
        got = np.frombuffer(out, np.uint32).reshape(n, 4)
        assert all((got[k] == want[k % 3]).all() for k in range(n))
        return 0

    default = WideFibProver.STREAM_SPIN_DEFAULT
    for bad, other in (streams, streams[::-1]):
        assert call(bad, 0) == ETIMEOUT
        sync(other.cuda_stream)
        assert call(other, default) == 0
        sync(bad.cuda_stream)
        assert call(bad, default) == 0
