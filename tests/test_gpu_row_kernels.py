"""Proofs at the edges of the composition's and the quotients' row kernels,
byte for byte as the oracle's."""
import pytest

from stwo_b200 import DeviceColumn, WideFibProver, wide_fib_config

pytestmark = pytest.mark.gpu


def check(oracle, log_n, cols, **options):
    a, b = oracle.wide_fib_inputs(log_n, 70 + cols)
    ref = oracle.prove_wide_fib(oracle.wide_fib_config(log_n, cols, **options), a, b)
    prover = WideFibProver(wide_fib_config(log_n, cols, **options))
    assert prover.prove(DeviceColumn.from_host(a), DeviceColumn.from_host(b)) == ref
    prover.close()


@pytest.mark.parametrize("log_n", [8, 9, 13])
@pytest.mark.parametrize("cols", [3, 5, 6, 7])
def test_few_columns(oracle, log_n, cols):
    # from 6 columns on the composition is taken on the tensor cores (2^9 points or more)
    check(oracle, log_n, cols)
