"""Proofs at the edges of the composition's and the quotients' row kernels,
byte for byte as the oracle's, and those with the longest decommitments."""
import hashlib
import json
import os

import numpy as np
import pytest

from stwo_b200 import DeviceColumn, WideFibProver, wide_fib_config

pytestmark = pytest.mark.gpu


def check(oracle, log_n, cols, **options):
    a, b = oracle.wide_fib_inputs(log_n, 70 + cols)
    ref = oracle.prove_wide_fib(oracle.wide_fib_config(log_n, cols, **options), a, b)
    prover = WideFibProver(wide_fib_config(log_n, cols, **options))
    assert prover.prove(DeviceColumn.from_host(a), DeviceColumn.from_host(b), cap=1 << 25) == ref
    prover.close()


@pytest.mark.parametrize("log_n", [8, 9, 13])
@pytest.mark.parametrize("cols", [3, 5, 6, 7])
def test_few_columns(oracle, log_n, cols):
    # from 6 columns on the composition is taken on the tensor cores (2^9 points or more)
    check(oracle, log_n, cols)


@pytest.mark.parametrize("log_n,cols", [(8, 128), (8, 129), (9, 120), (9, 121), (11, 160), (13, 300), (10, 1016)])
def test_many_columns(oracle, log_n, cols):
    # five and more weight stages of 32 columns, two blocks an SM and then one;
    # 1016 columns and the composition's 8 are as many as the operands hold
    check(oracle, log_n, cols)


@pytest.mark.parametrize("log_n", [9, 10, 15])
def test_long_decommitments(oracle, log_n):
    # 1016 columns at up to 4096 queries.  About 1.04e6, 1.8e6 and 4.5e6 words:
    # the plan and its words in page-locked memory (up to 1.4e6), staged in one
    # chunk, and in three chunks up and two down
    check(oracle, log_n, 1016, n_queries=4096)


def test_tile_bits_above_the_tables(oracle):
    # 2^24 quotient rows are 2^15 tiles; the tables of a tile's base point cover 14 bits
    r = np.random.default_rng(23)
    a, b = (r.integers(0, (1 << 31) - 1, 1 << 23, dtype=np.uint32) for _ in range(2))
    prover = WideFibProver(wide_fib_config(23, 3))
    got = prover.prove(DeviceColumn.from_host(a), DeviceColumn.from_host(b))
    prover.close()
    with open(os.path.join(os.path.dirname(__file__), "golden", "full_size_digests.json")) as f:
        want = json.load(f)
    assert (hashlib.sha256(got).hexdigest(), len(got)) == (want["wide_fib_narrow_sha256"], want["wide_fib_narrow_bytes"])
    assert oracle.verify_wide_fib(got, 23, 3) is None
