"""The row-wise setup stages at the edges of their size classes, against the
oracle (the reference's stages on the host), bit for bit."""
import numpy as np
import pytest

import thermofem_b200 as tf
from oracle import oracle as O
from conftest import to_device

pytestmark = pytest.mark.gpu


def random_matrix(rows, length, symmetric, seed):
    """About `length` entries per row (columns drawn near the row and far
    from it), full diagonal; a symmetric pattern or not; unsymmetric values."""
    rng = np.random.default_rng(seed)
    pattern = np.zeros((rows, rows), bool)
    for i in range(rows):
        k = max(0, min(rows, length + int(rng.integers(-1, 2))) - 1)
        near = rng.choice(rows, size=k, replace=False)
        pattern[i, near] = True
    if symmetric:
        pattern = np.triu(pattern, 1)
        pattern |= pattern.T
    np.fill_diagonal(pattern, True)
    off = np.concatenate([[0], pattern.sum(1).cumsum()]).astype(np.int32)
    idx = np.nonzero(pattern)[1].astype(np.int32)
    val = -np.exp(rng.standard_normal(idx.size))
    val[rng.random(idx.size) < 0.1] *= -1
    diag = np.repeat(np.arange(rows), np.diff(off)) == idx
    val[diag] = 4.0 * length
    return O.Csr(rows, off, idx, val)


def same(a, b):
    off, idx, val = a.host()
    return (np.array_equal(off, b.offsets) and np.array_equal(idx, b.indices) and
            np.array_equal(val.view(np.int64), np.asarray(b.values).view(np.int64)))


# merged rows of up to 32, 64, 128, 256 and 512 entries, and past 512 (the
# sort over all coordinates); row counts that divide by no tile
@pytest.mark.parametrize("length", [1, 2, 7, 9, 16, 17, 31, 33, 64, 65, 127, 129, 200])
@pytest.mark.parametrize("symmetric", [False, True])
def test_aggregates_and_coarse_operator(ctx, length, symmetric):
    for rows in (1, 5, 67, 331):
        a = O.canonical(random_matrix(rows, length, symmetric, 1000 * length + rows))
        da = to_device(a)
        g = O.strength(a, 0.25)
        dg = tf.strength(da, 0.25, ctx=ctx)
        assert same(dg, g)
        for rounds, absorb in ((1, True), (8, True), (8, False)):
            t = tf.aggregate(dg, rounds, absorb, ctx=ctx)
            ot = O.aggregate(g, rounds, absorb)
            assert np.array_equal(t.map.cpu().numpy(), ot.map)
            assert np.array_equal(t.offsets.cpu().numpy(), ot.offsets)
            assert np.array_equal(t.members.cpu().numpy(), ot.members)
            assert np.array_equal(t.histogram, ot.histogram)
            assert same(tf.galerkin(da, t, ctx=ctx), O.galerkin(a, ot.map, t.coarse_rows))
