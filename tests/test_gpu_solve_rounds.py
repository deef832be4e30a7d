"""The whole-solve graph's rounds of five iterations and the smoother on the
caller's own vectors give the bits of one launch after another."""
import numpy as np
import pytest
import torch

import thermofem_b200 as tf
from conftest import to_device
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


# a refresh inside a round, at its end, past several rounds and never;
# solves that stop before, at and after a round's end, and converge in one
@pytest.mark.parametrize("kind", ["Cg", "BiCgStab"])
@pytest.mark.parametrize("preconditioner", ["amg", "identity"])
@pytest.mark.parametrize("interval", [1, 3, 5, 7, 10, 50])
def test_rounds_match_single_iterations(ctx, kind, preconditioner, interval):
    m = P.laplace2d(31)
    n = len(m[0]) - 1
    b = torch.tensor(P.rhs_uniform(n, 17), device="cuda")
    for limit in (0, 1, 4, 5, 6, 9, 10, 11, 200):
        out = []
        for mode in (1, 0):
            s = getattr(tf, kind)(tf.solver_options(max_iterations=limit, residual_refresh_interval=interval),
                                  preconditioner, tf.amg_options(jacobi_weight=2 / 3), ctx=ctx)
            s.setup(to_device(m))
            s.set_graph_mode(mode)
            x = torch.zeros(n, dtype=torch.float64, device="cuda")
            out.append((s.apply(b, x), x))
        assert out[0][0] == out[1][0], limit
        assert torch.equal(out[0][1], out[1][1]), limit


def launched(a, dinv, b, x, weight, sweeps, ctx):
    for _ in range(sweeps):
        x = tf.jacobi_sweep(a, dinv, b, x, weight, ctx=ctx)
    return x


# a stencil (banded copy) and a matrix without one; vectors apart, the same,
# overlapping, off their 16-byte boundary and in host memory
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("sweeps", [1, 2, 3, 4])
@pytest.mark.parametrize("stencil", [True, False])
def test_smoother_on_any_vectors(ctx, dtype, sweeps, stencil):
    if stencil:
        m = P.convdiff3d(13, seed=5)
    else:
        rng = np.random.default_rng(4)
        dense = np.where(rng.random((301, 301)) < 0.05, rng.standard_normal((301, 301)), 0.0)
        np.fill_diagonal(dense, 40.0)
        m = (np.concatenate([[0], (dense != 0).sum(1).cumsum()]).astype(np.int32),
             np.nonzero(dense)[1].astype(np.int32), dense[dense != 0])
    n = len(m[0]) - 1
    a = to_device(m, dtype)
    dinv = tf.inverse_diagonal(a, ctx=ctx)
    smoother = tf.Jacobi(sweeps, 2 / 3, dtype=dtype, ctx=ctx)
    smoother.setup(a)
    b = torch.tensor(P.rhs_uniform(n, 3), device="cuda").to(dtype)
    x = torch.tensor(P.rhs_uniform(n, 4), device="cuda").to(dtype)
    want = launched(a, dinv, b, x, 2 / 3, sweeps, ctx)
    assert torch.equal(smoother.apply(b, x.clone()), want)
    room = torch.empty(2 * n + 3, dtype=dtype, device="cuda")
    off = room[1:n + 1].copy_(b), room[n + 2:2 * n + 2].copy_(x)
    assert torch.equal(smoother.apply(*off), want) and torch.equal(off[0], b)
    host = x.cpu()
    assert torch.equal(smoother.apply(b.cpu(), host), want.cpu())
    host = x.cpu()
    assert torch.equal(smoother.apply(b, host), want.cpu())
    same = x.clone()
    assert torch.equal(smoother.apply(same, same), launched(a, dinv, x, x, 2 / 3, sweeps, ctx))
    room = torch.tensor(P.rhs_uniform(n + 1, 6), device="cuda").to(dtype)
    want = launched(a, dinv, room[1:].clone(), room[:-1].clone(), 2 / 3, sweeps, ctx)
    assert torch.equal(smoother.apply(room[1:], room[:-1]), want)
