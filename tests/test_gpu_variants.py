"""Edges of the kernels' variants: sizes around a tile, a word or a chunk, and the calls that a
dispatch sends another way than their neighbours.  Integers are compared bitwise; the bars of
computed values are the ones of the path's own parity tests."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TWO_PI = 2 * np.pi


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def to_dev(a, dev):
    return torch.from_numpy(np.asfortranarray(a)).to(dev)


def relerr(got, want):
    return np.abs(np.asarray(got, dtype=np.float64) - want).max() / max(np.abs(want).max(), 1e-300)


@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 255, 257, 4097, 400_003])
def test_traversal_validation_counts_every_entry(gbg, dev, m):
    # the bitmap's word edges and the last, partial word; one entry named twice, one out of range
    rng = np.random.default_rng(m)
    perm = (rng.permutation(m) + 1).astype(np.int32)
    gbg.PointTraversalOrder(torch.from_numpy(perm).to(dev))
    for bad in (0, m + 1, -7):
        broken = perm.copy()
        broken[rng.integers(m)] = bad
        with pytest.raises(gbg.ArgumentError, match="1:%d, but it spans" % m):
            gbg.PointTraversalOrder(torch.from_numpy(broken).to(dev))
    if m > 1:
        twice = perm.copy()
        twice[0] = twice[m - 1]
        with pytest.raises(gbg.ArgumentError, match="names %d of %d" % (m - 1, m)):
            gbg.PointTraversalOrder(torch.from_numpy(twice).to(dev))
