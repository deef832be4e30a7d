"""A component's call has done its work on the GPU when it returns, whatever
is queued on the context's stream before it."""
import time

import pytest
import torch

import thermofem_b200 as tf
from conftest import to_device
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["sgd", "amg", "jacobi"])
def test_stream_is_idle_after_the_call(ctx, call):
    a = to_device(P.heat3d(8, seed=2))
    b = torch.tensor(P.rhs_uniform(a.rows, 3), device="cuda")
    x = torch.zeros_like(b)
    if call == "sgd":
        model = tf.Mlp(seed=3, ctx=ctx)
        f = tf.row_features(a, 0, ctx=ctx)
        run = lambda: (model.backward(f, torch.full((a.rows,), 0.7, device="cuda")), queue(), model.sgd(0.1))
    elif call == "amg":
        m = tf.Amg(tf.amg_options(hierarchy_type="f32"), ctx=ctx)
        m.setup(a)
        run = lambda: (queue(), m.apply(b, x))
    else:
        m = tf.Jacobi(ctx=ctx)
        m.setup(a)
        run = lambda: (queue(), m.apply(b, x))

    def queue():
        with torch.cuda.stream(ctx.stream):
            torch.cuda._sleep(200_000_000)  # 0.1 s and more

    for _ in range(3):  # an apply's first calls and its repeated one
        run()
        # (only the event that the wrapper records may follow the call's work)
        end = time.perf_counter() + 0.02
        while not ctx.stream.query() and time.perf_counter() < end:
            pass
        assert ctx.stream.query()
