"""Folds of two and three layers and lifted sums at word-aligned columns (the
general kernels) and at 16-byte aligned ones (whole loads), against the oracle."""
import numpy as np
import pytest

from oracle import ffi as oracle
from stwo_b200 import B200Backend, DeviceColumn, SecureColumn

pytestmark = pytest.mark.gpu
P = (1 << 31) - 1


class View:
    """n words of a column from word `at` on."""

    def __init__(self, words, at):
        self.col = DeviceColumn.from_host(np.concatenate([np.zeros(at, np.uint32), words]))
        self.ptr = self.col.ptr + 4 * at
        self.length = words.size
        self.log_size = words.size.bit_length() - 1


def column(log, seed, at):
    w = np.random.default_rng(seed).integers(0, P + 1, (4, 1 << log), dtype=np.uint32)  # P itself too
    return SecureColumn([View(c, at) for c in w]), list(w)


@pytest.mark.parametrize("at", [0, 1, 2, 4])
@pytest.mark.parametrize("step,log", [(2, 2), (2, 3), (2, 11), (2, 17), (3, 3), (3, 4), (3, 12), (3, 18)])
def test_fold_line_steps(step, log, at):
    be = B200Backend()
    init, lg = oracle.canonic_half_coset_root(20)
    tree = be.precompute_twiddles(init, lg)
    _, itw = oracle.precompute_twiddles(init, lg)
    col, w = column(log, 7 * log + step, at)
    alpha = np.random.default_rng(log).integers(0, P, 4, dtype=np.uint32)
    got = be.fold_line(col, alpha, tree, step).to_host()
    for a, b in zip(got, oracle.fold_line(w, itw, alpha, step)):
        assert (a == b).all()


@pytest.mark.parametrize("at", [0, 1, 2, 4])
@pytest.mark.parametrize("logs", [[1], [2], [5], [1, 2], [1, 3], [2, 3, 4, 5], [1, 9], [3, 4, 11, 17], [16, 17]])
def test_lifted_sums(logs, at):
    be = B200Backend()
    cols = [column(g, 50 + g, at) for g in logs]
    ref = oracle.lift_and_accumulate([w for _, w in cols])
    for a, b in zip(be.lift_and_accumulate([c for c, _ in cols]).to_host(), ref):
        assert (a == b).all()
