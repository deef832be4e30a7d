"""Components may be destroyed after their context: each destroy call succeeds
and the memory goes back to the device."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

SCRIPT = """
import sys; sys.path.insert(0, {root!r})
import ctypes as C, torch, thermofem_b200 as tf
from thermofem_b200 import problems as P
torch.zeros(1, device="cuda")
lib = tf.lib()
class Own(tf.Context):
    "a context with a stream of the library's own, destroyed with it"
    def __init__(self):
        self.device, h = 0, C.c_void_p()
        tf.check(lib.tf_ctx_create(0, None, C.byref(h)))
        self.h = h
        self.stream = torch.cuda.ExternalStream(lib.tf_ctx_stream(h))
def used():
    torch.cuda.synchronize(); torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free
def components(ctx, side):
    a = tf.DeviceCsr.from_host(*P.heat3d(side))
    amg, jacobi = tf.Amg(tf.amg_options(), ctx=ctx), tf.Jacobi(ctx=ctx)
    solvers = [tf.Cg(tf.solver_options(), "amg", tf.amg_options(hierarchy_type="f32"), ctx=ctx) for _ in range(2)]
    for c in [amg, jacobi] + solvers: c.setup(a)
    view = amg.level_matrix(0)
    batch, mlp = tf.Batch(solvers, ctx=ctx), tf.Mlp(ctx=ctx)
    b = torch.ones(a.rows, dtype=torch.float64, device="cuda")
    amg.apply(b); jacobi.apply(b, b.clone()); batch.apply([b, b], [torch.zeros_like(b), torch.zeros_like(b)])
    return [("batch", batch)] + [("solver", s) for s in solvers] + [("amg", amg), ("jacobi", jacobi), ("mlp", mlp)]
def destroy(parts):
    for name, c in parts:
        rc = getattr(lib, "tf_" + name + "_destroy")(c.h)
        assert rc == 0, (name, rc, lib.tf_last_error())
        c.h = None
for kind in (Own, lambda: tf.Context(0)):
    ctx = kind(); destroy(components(ctx, 16)); ctx.close()
base = used()
for kind in (Own, lambda: tf.Context(0)):
    ctx = kind()
    parts = components(ctx, 80)  # 0.5 GiB and more
    ctx.close()
    destroy(parts)
    left = used() - base
    assert left <= 64 << 20, left
    # another context alive, as free memory of the size of the closed one's may be in use again
    ctx, other = kind(), kind()
    parts = components(ctx, 24)
    ctx.close()
    third = kind()
    destroy(parts)
    destroy(components(third, 12)); destroy(components(other, 12))
    third.close(); other.close()
    left = used() - base
    assert left <= 64 << 20, left
print("ok")
"""


@pytest.mark.gpu
def test_components_outlive_their_context():
    # (freed host memory is overwritten, so that nobody reads a closed context unnoticed)
    env = dict(os.environ, MALLOC_PERTURB_="90", GLIBC_TUNABLES="glibc.malloc.tcache_count=0")
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT)], capture_output=True, text=True, timeout=300,
                       env=env)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
