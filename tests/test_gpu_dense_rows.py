"""Small levels with a dense row among short ones: the small-level region (one
CTA over its image, a cluster of one or more CTAs) gives the bits of launched
levels."""
import numpy as np
import pytest
import torch

import thermofem_b200 as tf
from conftest import to_device
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


def arrow(n, bands, seed):
    """Dense first row and column, `bands` couplings to either side."""
    rng = np.random.default_rng(seed)
    a = np.zeros((n, n))
    a[0, 1:] = -1 - rng.random(n - 1)
    for q in range(1, bands + 1):
        a[np.arange(1, n - q), np.arange(1 + q, n)] = -1 - rng.random(n - 1 - q)
    a = np.triu(a, 1)
    a += a.T
    np.fill_diagonal(a, 0.5 - a.sum(1))
    keep = a != 0
    off = np.concatenate([[0], keep.sum(1).cumsum()]).astype(np.int32)
    return off, np.nonzero(keep)[1].astype(np.int32), a[keep]


# no bands: hardly any contraction, 20 levels (V and F only: a W-cycle visits
# the last 2^19 times)
@pytest.mark.parametrize("hierarchy", ["f32", "f64", "f32v"])
@pytest.mark.parametrize("n,bands,cycles", [(70, 0, "vf"), (200, 0, "vf"), (200, 1, "v"), (333, 2, "vwf"), (1100, 2, "vwf"),
                                            (1500, 4, "vwf"), (4000, 3, "v")])
def test_region_matches_launched_levels(ctx, n, bands, cycles, hierarchy):
    a = to_device(arrow(n, bands, n + bands))
    b = torch.tensor(P.rhs_uniform(n, 3), device="cuda")
    for cycle in cycles:
        out = []
        for region in (1200, 0):
            amg = tf.Amg(tf.amg_options(cycle=cycle, hierarchy_type=hierarchy, jacobi_weight=2 / 3, coarse_rows=16,
                                        small_level_rows=region), ctx=ctx)
            amg.setup(a)
            out.append([amg.apply(b) for _ in range(3)])
        assert bool(torch.isfinite(out[0][0]).all())
        for x in out[0] + out[1]:
            assert torch.equal(x, out[0][0]), cycle
