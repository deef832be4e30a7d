"""Small operators: the wide sliced kernel (whole slices in flight), the
launch shapes taken by rule, and the one-CTA region over them give the bits of
the row-tile kernels and of separately launched levels."""
import numpy as np
import pytest
import torch

import thermofem_b200 as tf
from conftest import to_device
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


def ragged(n, longest, seed):
    """A graph Laplacian with rows of 1 to about `longest` entries, some rows
    of the diagonal alone."""
    rng = np.random.default_rng(seed)
    a = np.zeros((n, n))
    for i in range(0, n - 1, 2):
        k = int(rng.integers(1, max(2, longest // 2 + 1)))
        for j in rng.integers(0, n - n // 16, size=k):
            if i != j and i < n - n // 16:
                a[i, j] = a[j, i] = -np.exp(rng.standard_normal())
    np.fill_diagonal(a, 0.25 - a.sum(1))
    pattern = a != 0
    off = np.concatenate([[0], pattern.sum(1).cumsum()]).astype(np.int32)
    return off, np.nonzero(pattern)[1].astype(np.int32), a[pattern]


# row counts around slices and tiles; slices of up to 24 slots (one batch of
# the wide kernel), just more, and several batches
@pytest.mark.parametrize("hierarchy", ["f32", "f64", "f32v"])
@pytest.mark.parametrize("cycle", ["v", "w", "f"])
@pytest.mark.parametrize("n,longest", [(33, 4), (257, 8), (513, 24), (700, 26), (1500, 60), (2049, 160)])
def test_small_levels_give_identical_cycles(ctx, hierarchy, cycle, n, longest, monkeypatch):
    a = to_device(ragged(n, longest, 10 * n + longest))
    b = torch.tensor(P.rhs_uniform(n, 7), device="cuda")
    out = []
    for sliced, region in (("1", 1200), ("1", 0), ("0", 0), ("0", 1200)):
        monkeypatch.setenv("THERMOFEM_B200_SLICED", sliced)
        amg = tf.Amg(tf.amg_options(cycle=cycle, hierarchy_type=hierarchy, jacobi_weight=2 / 3, coarse_rows=16,
                                    small_level_rows=region), ctx=ctx)
        amg.setup(a)
        out.append(amg.apply(b))
    assert bool(torch.isfinite(out[0]).all())
    for other in out[1:]:
        assert torch.equal(out[0], other)


@pytest.mark.parametrize("hierarchy", ["f32", "f64"])
def test_small_levels_give_identical_solves(ctx, hierarchy, monkeypatch):
    m = P.heat3d(27, seed=91)
    n = len(m[0]) - 1
    b = torch.tensor(P.rhs_uniform(n, 92), device="cuda")
    out = []
    for sliced in ("1", "0"):
        monkeypatch.setenv("THERMOFEM_B200_SLICED", sliced)
        s = tf.Cg(tf.solver_options(), "amg", tf.amg_options(hierarchy_type=hierarchy, jacobi_weight=2 / 3), ctx=ctx)
        s.setup(to_device(m))
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        out.append((s.apply(b, x), x))
    assert out[0][0] == out[1][0] and torch.equal(out[0][1], out[1][1])
