"""A level's arrays and checks in one pass, at the row lengths where the number
of lanes per row changes: the operator the cycle streams, its diagonal, and
each reason to refuse it."""
import numpy as np
import pytest
import torch

import thermofem_b200 as tf
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


def circulant(n, length):
    """`length` entries a row: a dominant diagonal and neighbours on a ring
    (columns up to n - 1 rows away)."""
    shifts = np.array([0] + [s for k in range(1, length) for s in (k, -k)][:length - 1])
    idx = np.sort((np.arange(n)[:, None] + shifts[None, :]) % n, axis=1)
    rng = np.random.default_rng(n + length)
    val = -1.0 - rng.random(idx.shape)
    val[idx == np.arange(n)[:, None]] = 4.0 * length
    off = np.arange(n + 1, dtype=np.int32) * length
    return off, idx.reshape(-1).astype(np.int32), val.reshape(-1)


def device(off, idx, val):
    return tf.DeviceCsr.from_host(off, idx, val)


def amg(ctx, hierarchy, **kw):
    return tf.Amg(tf.amg_options(hierarchy_type=hierarchy, jacobi_weight=2 / 3, **kw), ctx=ctx)


# lanes change at mean row lengths between these; 33,000 rows need 4-byte columns
@pytest.mark.parametrize("hierarchy", ["f32", "f64", "f32v"])
@pytest.mark.parametrize("n,length", [(33, 1), (33, 2), (257, 3), (257, 5), (300, 16), (301, 33), (401, 70), (33000, 5)])
def test_operator_and_diagonal(ctx, hierarchy, n, length):
    off, idx, val = circulant(n, length)
    m = amg(ctx, hierarchy, max_levels=1, coarse_lu_rows=1, coarse_sweeps=1)
    m.setup(device(off, idx, val))
    cycle = torch.float32 if hierarchy == "f32" else torch.float64
    stored = torch.tensor(val, device="cuda")
    if hierarchy != "f64":
        stored = stored.float()
    x = torch.tensor(P.rhs_uniform(n, 5), device="cuda").to(cycle)
    a = tf.DeviceCsr(torch.tensor(off, device="cuda"), torch.tensor(idx, device="cuda"), stored.to(cycle))
    assert torch.equal(m.level_spmv(0, x), tf.spmv(a, x, ctx=ctx))
    # one sweep from zero: w D^-1 b
    b = torch.tensor(P.rhs_uniform(n, 6), device="cuda")
    want = tf.jacobi_zero(tf.inverse_diagonal(a, ctx=ctx), b.to(cycle), 2 / 3, ctx=ctx)
    assert torch.equal(m.apply(b), want.double())


@pytest.mark.parametrize("hierarchy", ["f32", "f64", "f32v"])
@pytest.mark.parametrize("row", [0, 130, 256])
@pytest.mark.parametrize("bad,refused", [("zero", "all"), ("missing", "all"), ("subnormal reciprocal", "all"),
                                         ("below f32", "f32"), ("above f32", "f32")])
def test_refused_diagonals(ctx, hierarchy, row, bad, refused):
    off, idx, val = circulant(257, 5)
    at = np.flatnonzero((np.repeat(np.arange(257), 5) == idx) & (idx == row))[0]
    if bad == "missing":
        keep = np.arange(idx.size) != at
        off = (off - (np.arange(258) > row)).astype(np.int32)
        idx, val = idx[keep], val[keep]
    else:
        val[at] = {"zero": 0.0, "subnormal reciprocal": 1e-320, "below f32": 1e-60, "above f32": 1e60}[bad]
    m = amg(ctx, hierarchy)
    if refused == "all" or hierarchy != "f64":
        with pytest.raises(tf.InvalidArgument, match="diagonal"):
            m.setup(device(off, idx, val))
    else:
        m.setup(device(off, idx, val))
