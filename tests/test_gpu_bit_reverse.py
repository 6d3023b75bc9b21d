"""Bit reversal at the edges of its two kernels (word swaps below 2^10 words,
32 x 32-word tiles from there): self-paired and paired tiles, in and out of
place, columns at any word alignment."""
import numpy as np
import pytest

from stwo_b200 import B200Backend, DeviceColumn

pytestmark = pytest.mark.gpu
P = (1 << 31) - 1


class View:
    """A column `offset` words into a larger buffer."""

    def __init__(self, buf, offset, log_size):
        self.buf, self.ptr, self.log_size = buf, buf.ptr + 4 * offset, log_size


@pytest.mark.parametrize("log_n", [9, 10, 11, 12, 15, 19])
@pytest.mark.parametrize("in_place", [False, True])
def test_bit_reverse_edges(oracle, log_n, in_place):
    be = B200Backend()
    r = np.random.default_rng(log_n)
    n, gap = 1 << log_n, 3
    vals = [r.integers(0, P + 1, n, dtype=np.uint32) for _ in range(3)]
    host = np.zeros(3 * (n + gap) + 1, np.uint32)
    for k, v in enumerate(vals):
        host[1 + k * (n + gap):1 + k * (n + gap) + n] = v
    src = DeviceColumn.from_host(host)
    dst = src if in_place else DeviceColumn.from_host(np.zeros_like(host))
    views = [[View(b, 1 + k * (n + gap), log_n) for k in range(3)] for b in (src, dst)]
    be.bit_reverse_columns(views[0], None if in_place else views[1])
    want = np.zeros_like(host)
    for k, v in enumerate(vals):
        want[1 + k * (n + gap):1 + k * (n + gap) + n] = oracle.bit_reverse(v)
    assert (dst.to_host() == want).all()  # the words between the columns too
    if not in_place:
        assert (src.to_host() == host).all()
    be.bit_reverse_column(views[1][1])
    want[1 + n + gap:1 + n + gap + n] = vals[1]
    assert (dst.to_host() == want).all()
