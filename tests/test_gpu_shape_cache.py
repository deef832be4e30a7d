"""Launch shapes of a caller's CSR arrays and of a component's copy of the same
operator do not replace each other, in whatever order they are tuned."""
import numpy as np
import pytest
import torch

import thermofem_b200 as tf
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


def box(nx, ny, nz):
    """7-point Laplacian plus identity; columns nx ny rows away."""
    n = nx * ny * nz
    i = np.arange(n)
    ix, iy, iz = i % nx, i // nx % ny, i // (nx * ny)
    steps = np.array([-nx * ny, -nx, -1, 0, 1, nx, nx * ny])
    keep = np.stack([iz > 0, iy > 0, ix > 0, ix >= 0, ix < nx - 1, iy < ny - 1, iz < nz - 1], 1)
    off = np.concatenate([[0], keep.sum(1).cumsum()]).astype(np.int32)
    return off, (i[:, None] + steps)[keep].astype(np.int32), np.broadcast_to(np.where(steps == 0, 7.0, -1.0), keep.shape)[keep]


# beyond 2-byte columns (the banded copy then stands beside 4-byte ones, as in
# the caller's arrays), under and over the rows from which shapes are timed
@pytest.mark.parametrize("nx,ny,nz", [(182, 183, 4), (190, 190, 9)])
@pytest.mark.parametrize("dtype,hierarchy", [("f64", "f64"), ("f32", "f32")])
def test_copy_is_streamed_whenever_the_caller_tunes(ctx, nx, ny, nz, dtype, hierarchy):
    t = {"f64": torch.float64, "f32": torch.float32}[dtype]
    a = tf.DeviceCsr.from_host(*box(nx, ny, nz), dtype=t)
    x = torch.tensor(P.rhs_uniform(a.rows, 3), device="cuda").to(t)
    want = tf.spmv(a, x, ctx=ctx)
    smoother = tf.Jacobi(2, 2 / 3, dtype=t, ctx=ctx)
    swept = x.clone()
    dinv = tf.inverse_diagonal(a, ctx=ctx)
    for _ in range(2):
        swept = tf.jacobi_sweep(a, dinv, x, swept, 2 / 3, ctx=ctx)
    for order in ("caller", "component", "caller"):
        if order == "caller":
            tf.autotune_spmv(a, x, ctx=ctx)
        s = tf.Cg(tf.solver_options(t), "amg", tf.amg_options(hierarchy_type=hierarchy), dtype=t, ctx=ctx)
        s.setup(a)
        smoother.setup(a)
        if order == "component":
            tf.autotune_spmv(a, x, ctx=ctx)
        assert s.spmv_layout()[0] == "banded" and s.level_spmv_layout(0)[0] == "banded"
        assert torch.equal(s.spmv(x), want) and torch.equal(tf.spmv(a, x, ctx=ctx), want)
        assert torch.equal(smoother.apply(x, x.clone()), swept)
        tf.set_spmv_config(a, 2, 2, 100, 1, ctx=ctx)
        assert s.spmv_layout()[0] == "banded"
        del s
