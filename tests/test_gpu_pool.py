"""The device memory pool: free memory is kept within its bound while a
context lives and given back with the device's last one; components may
outlive their context's use of it in any destruction order."""
import subprocess
import sys

import pytest

from conftest import ROOT

SCRIPT = """
import sys; sys.path.insert(0, {root!r})
import torch, thermofem_b200 as tf
from thermofem_b200 import problems as P
torch.cuda.init(); torch.zeros(1, device="cuda")
def used():
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free
def work(ctx, m, hierarchy):
    a = tf.DeviceCsr.from_host(*P.heat3d(m))
    s = tf.Cg(tf.solver_options(), "amg", tf.amg_options(hierarchy_type=hierarchy), ctx=ctx)
    s.setup(a)
    b = torch.ones(a.rows, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    assert s.apply(b, x)["status"] == "Converged"
    return s, x
ctx = tf.Context(0)
s, x0 = work(ctx, 40, "f32")
del s
ctx.close()
base = used()
ctx, other = tf.Context(0), tf.Context(0)
first, x1 = work(ctx, 40, "f32")
second, x2 = work(other, 96, "f64")
assert torch.equal(x0, x1)
del second
held = used() - base
assert held <= (4 << 30) + (1 << 30), held
third, x3 = work(other, 40, "f32")
assert torch.equal(x0, x3)
del first, third, x1, x2, x3
ctx.close()
other.close()
left = used() - base
assert left <= 64 << 20, left
print("ok", held, left)
"""


@pytest.mark.gpu
def test_pool_memory_is_bounded_and_given_back():
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
