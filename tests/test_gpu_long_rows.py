"""Launch shapes and copies by the mean row length: every class of the rule
gives the bits of the row tiles, alone and in whole cycles."""
import numpy as np
import pytest
import torch

import thermofem_b200 as tf
from conftest import to_device
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


def ragged(n, mean, seed):
    """A symmetric graph Laplacian plus a mass term with rows of about `mean`
    entries (half to one and a half times that) near the diagonal."""
    rng = np.random.default_rng(seed)
    degree = rng.integers(max(1, mean // 4), max(2, 3 * mean // 4), n)
    src = np.repeat(np.arange(n), degree)
    dst = (src + rng.integers(1, min(n - 1, 4 * mean) + 1, src.size)) % n
    edge = np.unique(np.stack([np.minimum(src, dst), np.maximum(src, dst)], 1)[src != dst], axis=0)
    w = np.exp(rng.standard_normal(len(edge)))
    a, b = edge[:, 0], edge[:, 1]
    diag = 0.25 + np.bincount(a, w, n) + np.bincount(b, w, n)
    r, c = np.concatenate([a, b, np.arange(n)]), np.concatenate([b, a, np.arange(n)])
    v = np.concatenate([-w, -w, diag])
    order = np.lexsort((c, r))
    off = np.concatenate([[0], np.bincount(r, minlength=n).cumsum()]).astype(np.int32)
    return off, c[order].astype(np.int32), v[order]


# (rows, mean): around the row lengths where the rule changes (16, 24, 40, 80,
# 100, 128, 200 entries), the rows that do (512, 8,192, 65,536), and past 4M
# entries (timed)
SIZES = [(300, 13), (2049, 17), (700, 30), (90, 46), (513, 60), (8191, 50), (8300, 50), (300, 90), (600, 120), (1025, 190),
         (1300, 230), (400, 260), (66000, 46), (24000, 180)]


@pytest.mark.parametrize("hierarchy", ["f32", "f64", "f32v"])
@pytest.mark.parametrize("rows,mean", SIZES)
def test_cycles_and_products(ctx, rows, mean, hierarchy, monkeypatch):
    m = ragged(rows, mean, rows + mean)
    a = to_device(m)
    b = torch.tensor(P.rhs_uniform(rows, 5), device="cuda")
    cycle = torch.float32 if hierarchy == "f32" else torch.float64
    out = []
    for sliced in ("1", "0"):
        monkeypatch.setenv("THERMOFEM_B200_SLICED", sliced)
        got = []
        for kind in ("v", "w"):
            amg = tf.Amg(tf.amg_options(cycle=kind, hierarchy_type=hierarchy, jacobi_weight=2 / 3, small_level_rows=0),
                         ctx=ctx)
            amg.setup(a)
            got.append(amg.apply(b))
        for d in range(amg.level_count()):
            n = amg.level_statistics()[d]["rows"]
            x = torch.tensor(P.rhs_uniform(n, 6 + d), device="cuda").to(cycle)
            got.append(amg.level_spmv(d, x))
        out.append(got)
    assert bool(torch.isfinite(out[0][0]).all())
    for u, v in zip(*out):
        assert torch.equal(u, v)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("rows,mean", SIZES)
def test_solver_operator(ctx, rows, mean, dtype):
    t = torch.float32 if dtype == "f32" else torch.float64
    a = to_device(ragged(rows, mean, rows + mean), t)
    x = torch.tensor(P.rhs_uniform(rows, 7), device="cuda").to(t)
    s = tf.Cg(tf.solver_options(t), "identity", dtype=t, ctx=ctx)
    want = tf.spmv(a, x, ctx=ctx)
    s.setup(a)
    assert torch.equal(s.spmv(x), want) and torch.equal(tf.spmv(a, x, ctx=ctx), want)
