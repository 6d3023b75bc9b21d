"""Node levels in one launch: trees at the edges of a block's subtree (2^8
hashes), of what the last block stages (2^17 in all) and of the several-levels-
a-thread kernel (2^18 up), against the oracle; trees of two streams at once."""
import numpy as np
import pytest

from oracle import ffi as oracle
from stwo_b200 import B200Backend, DeviceBuffer, DeviceColumn, layer_to_host, sync

pytestmark = pytest.mark.gpu
P = (1 << 31) - 1


def words(log, seed):
    return np.random.default_rng(seed).integers(0, P, 1 << log, dtype=np.uint32)


@pytest.mark.parametrize("log", [1, 2, 7, 8, 9, 10, 16, 17, 18, 19, 20])
@pytest.mark.parametrize("m31", [False, True])
def test_layers(log, m31):
    be = B200Backend()
    w = words(log, log)
    layers = be.build_merkle_layers([DeviceColumn.from_host(w)], log, m31)
    ref = oracle.merkle_build_layers([w], log, m31)
    for k in range(log + 1):
        assert (layer_to_host(layers[k]) == ref[k]).all(), k
    own = [DeviceBuffer(32 << k) for k in range(log)] + [layers[log]]
    for b in own[:-1]:
        b.upload(np.full(b.nbytes, 0xFF, np.uint8))
    be.build_nodes(own, m31)
    assert all((layer_to_host(own[k]) == ref[k]).all() for k in range(log))
    if log > 1:
        assert (layer_to_host(be.build_next_layer(layers[log], m31)) == ref[log - 1]).all()


def test_two_streams():
    import torch
    streams = [torch.cuda.Stream() for _ in range(2)]
    bes = [B200Backend(s.cuda_stream) for s in streams]
    w = [words(16, 90 + k) for k in range(2)]
    cols = [DeviceColumn.from_host(x) for x in w]
    ref = [oracle.merkle_build_layers([x], 16, False) for x in w]
    for _ in range(8):
        got = [bes[k].build_merkle_layers([cols[k]], 16) for k in range(2)]
        for k in range(2):
            sync(streams[k].cuda_stream)
            assert all((layer_to_host(got[k][j]) == ref[k][j]).all() for j in range(17))
