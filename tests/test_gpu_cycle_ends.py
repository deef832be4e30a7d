"""A cycle whose first and last step work on the caller's vectors gives the
bits of one with conversions before and after it."""
import pytest
import torch

import thermofem_b200 as tf
from conftest import to_device
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


# every number of sweeps that decides what the first and the last step are;
# a finest level above and below the size that prolongs inside its sweep
@pytest.mark.parametrize("hierarchy", ["f32", "f64", "f32v"])
@pytest.mark.parametrize("cycle", ["v", "w", "f"])
@pytest.mark.parametrize("pre,post", [(1, 1), (2, 2), (0, 1), (1, 0), (3, 1), (0, 0)])
@pytest.mark.parametrize("side", [3, 11, 54])
def test_apply_matches_separate_conversions(ctx, hierarchy, cycle, pre, post, side, monkeypatch):
    a = to_device(P.heat3d(side, seed=3))
    n = a.rows
    b = torch.tensor(P.rhs_uniform(n, 8), device="cuda")
    out = []
    for fuse in ("1", "0"):
        monkeypatch.setenv("THERMOFEM_B200_FUSE", fuse)
        amg = tf.Amg(tf.amg_options(cycle=cycle, hierarchy_type=hierarchy, jacobi_weight=2 / 3, pre_sweeps=pre,
                                    post_sweeps=post), ctx=ctx)
        amg.setup(a)
        out.append(amg.apply(b))
        room = torch.empty(n + 1, dtype=b.dtype, device="cuda")
        room[1:].copy_(b)
        for _ in range(2):  # in place, off a 16-byte boundary, repeated
            again = amg.apply(room[1:], room[1:])
            assert torch.equal(again, out[-1])
            room[1:].copy_(b)
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("hierarchy", ["f32", "f64"])
def test_single_precision_vectors(ctx, hierarchy, monkeypatch):
    a = to_device(P.heat3d(12, seed=4), torch.float32)
    b = torch.tensor(P.rhs_uniform(a.rows, 9), device="cuda").float()
    out = []
    for fuse in ("1", "0"):
        monkeypatch.setenv("THERMOFEM_B200_FUSE", fuse)
        amg = tf.Amg(tf.amg_options(hierarchy_type=hierarchy, jacobi_weight=2 / 3), dtype=torch.float32, ctx=ctx)
        amg.setup(a)
        out.append(amg.apply(b))
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("hierarchy", ["f32", "f64"])
def test_vectors_in_host_memory(ctx, hierarchy):
    a = to_device(P.heat3d(11, seed=5))
    b = torch.tensor(P.rhs_uniform(a.rows, 10))
    amg = tf.Amg(tf.amg_options(hierarchy_type=hierarchy, jacobi_weight=2 / 3), ctx=ctx)
    amg.setup(a)
    want = amg.apply(b.cuda()).cpu()
    host, x = b.pin_memory(), torch.zeros_like(b).pin_memory()
    for rhs, out in ((host, x), (b.cuda(), x), (host, torch.zeros_like(b, device="cuda"))):
        x.zero_()
        assert torch.equal(amg.apply(rhs, out).cpu(), want)
