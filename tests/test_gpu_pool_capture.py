"""Calls that use temporary arrays stay capturable while the memory pool gives
back what exceeds its bound."""
import pytest
import torch

import thermofem_b200 as tf

pytestmark = pytest.mark.gpu


# a scan of one launch and of three (with a temporary array of its own); the
# pool within its bound at the end of the captured call, and above it:
# temporaries of 4.8 GB, freed but not yet drained when the capture begins
@pytest.mark.parametrize("n", [1000, 3_000_000])
@pytest.mark.parametrize("above", [False, True])
def test_scan_inside_a_capture(ctx, n, above):
    x = torch.ones(n, dtype=torch.int32, device="cuda")
    want = tf.scan_exclusive(x, ctx=ctx)
    keys = torch.zeros(300_000_000 if above else 1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    kept = tf.radix_sort_pairs(keys, keys.view(torch.float64), end_bit=16, ctx=ctx)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = tf.scan_exclusive(x, ctx=ctx)
    for k in (1, 3):
        x.fill_(k)
        graph.replay()
        assert torch.equal(out, k * want)
    del kept
