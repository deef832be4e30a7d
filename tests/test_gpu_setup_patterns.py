"""Hierarchies of operators that no stencil gives, level by level against the
oracle: strong edges without an entry for their other direction (the sorted
strength graph), and ragged symmetric patterns (weights on the operator's own
pattern), with one, four and 32 lanes to a row and on both sides of the size
that one CTA aggregates (4,096 rows, 65,536 entries)."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import thermofem_b200 as tf
from conftest import to_device
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def operator(rows, length, pattern, seed):
    """About `length` entries a row near the diagonal and some far from it,
    unsymmetric values; pattern: symmetric, one-sided (a third of the edges
    have one direction only), upper (all of them) or sparse one-sided (one
    edge of the whole operator)."""
    rng = np.random.default_rng(seed)
    m = max(1, (length - 1) // 2)
    src = np.repeat(np.arange(rows), rng.integers(1, 2 * m, rows) if m > 1 else 1)
    dst = (src + rng.integers(1, max(2, min(rows, 8 * length)), src.size)) % rows
    far = rng.random(src.size) < 0.02
    dst[far] = rng.integers(0, rows, far.sum())
    lo, hi = np.minimum(src, dst), np.maximum(src, dst)
    edge = np.unique(np.stack([lo, hi], 1)[lo != hi], axis=0)
    lo, hi = edge[:, 0], edge[:, 1]
    both = {"symmetric": np.ones(lo.size, bool), "one-sided": rng.random(lo.size) < 0.67,
            "upper": np.zeros(lo.size, bool), "sparse": np.arange(lo.size) != lo.size // 2}[pattern]
    r, c = np.concatenate([lo, hi[both]]), np.concatenate([hi, lo[both]])
    v = -np.exp(rng.standard_normal(r.size))
    if pattern == "sparse":
        v[lo.size // 2] *= 1e3  # strong
    a = sp.csr_matrix((v, (r, c)), shape=(rows, rows))
    a = (a + sp.diags(0.5 + abs(a).sum(1).A1 + abs(a).sum(0).A1)).tocsr()
    a.sort_indices()
    return O.Csr(rows, a.indptr.astype(np.int32), a.indices.astype(np.int32), a.data)


def test_operators_have_the_lanes_meant():
    for length, lanes in ((3, 1), (9, 4), (60, 32)):
        a = operator(2000, length, "symmetric", length)
        mean = a.nnz // a.rows
        assert lanes == (1 if mean < 4 else (4 if mean < 24 else 32)), (length, mean)


@pytest.mark.parametrize("pattern", ["symmetric", "one-sided", "upper", "sparse"])
@pytest.mark.parametrize("rows,length", [(1, 3), (7, 3), (331, 3), (331, 9), (331, 60), (4096, 3), (4096, 9), (3001, 60),
                                         (4097, 3), (4097, 9), (4097, 60), (20011, 9)])
@pytest.mark.parametrize("absorb", [True, False])
def test_hierarchy_matches_oracle(ctx, pattern, rows, length, absorb):
    if rows == 1 and pattern != "symmetric":
        pytest.skip("one row has no edges")
    a = operator(rows, length, pattern, rows + length)
    opts = dict(coarse_rows=16, matching_rounds=8 if absorb else 2, absorb_singletons=absorb)
    amg = tf.Amg(tf.amg_options(**opts), dtype=torch.float64, ctx=ctx)
    amg.setup(to_device(a))
    ora = O.Amg(a, **opts)
    assert amg.level_count() == ora.levels
    assert (amg.stop_reason(), amg.coarse_solver()) == (ora.stop_reason(), ora.coarse_solver())
    stats = amg.level_statistics()
    for d in range(ora.levels):
        r, z, hist = ora.level_info(d)
        assert (stats[d]["rows"], stats[d]["nonzeros"], stats[d]["aggregate_sizes"]) == (r, z, hist.tolist())
        off, idx, val = amg.level_matrix(d).host()
        want = ora.matrix(d)
        assert np.array_equal(off, want.offsets) and np.array_equal(idx, want.indices)
        assert np.array_equal(val.view(np.int64), want.values.view(np.int64))
        if d + 1 < ora.levels:
            mp, offs, mem, _ = amg.level_transfer(d)
            mp = mp.cpu().numpy()
            assert np.array_equal(mp, ora.map(d))
            assert np.array_equal(mem.cpu().numpy(), np.argsort(mp, kind="stable"))
            assert np.array_equal(np.diff(offs.cpu().numpy()), np.bincount(mp))
