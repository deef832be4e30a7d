"""The smoother takes vectors at any byte address of device memory, as its
copies in and out always did."""
import ctypes as C

import pytest
import torch

import thermofem_b200 as tf
from conftest import to_device
from thermofem_b200 import check, lib
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("sweeps", [1, 2, 3])
@pytest.mark.parametrize("rhs_at,x_at", [(1, 0), (0, 2), (3, 3), (4, 0), (0, 4), (4, 4), (8, 8)])
def test_vectors_at_any_byte(ctx, dtype, sweeps, rhs_at, x_at):
    a = to_device(P.convdiff3d(9, seed=6), dtype)
    n = a.rows
    m = tf.Jacobi(sweeps, 2 / 3, dtype=dtype, ctx=ctx)
    m.setup(a)
    b = torch.tensor(P.rhs_uniform(n, 7), device="cuda").to(dtype)
    x = torch.tensor(P.rhs_uniform(n, 8), device="cuda").to(dtype)
    want = m.apply(b, x.clone())
    size = n * b.element_size()

    def room(v, at):
        raw = torch.zeros(size + 16, dtype=torch.uint8, device="cuda")
        raw[at:at + size] = v.view(torch.uint8)
        return raw

    rb, rx = room(b, rhs_at), room(x, x_at)
    with ctx:
        check(lib().tf_jacobi_apply(m.h, C.c_void_p(rb.data_ptr() + rhs_at), C.c_void_p(rx.data_ptr() + x_at)))
    got = rx[x_at:x_at + size].clone().view(dtype)
    assert torch.equal(got, want)
    assert torch.equal(rb, room(b, rhs_at))
    assert not rx[:x_at].any() and not rx[x_at + size:].any()
