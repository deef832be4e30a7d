"""Solves of a few iterations: the whole-solve graph gives what single
iterations give, and does not run a round of them past the end."""
import pytest
import torch

import thermofem_b200 as tf
from conftest import to_device
from thermofem_b200 import problems as P

pytestmark = pytest.mark.gpu


def solver(ctx, kind, m, mode=1, **kw):
    s = getattr(tf, kind)(tf.solver_options(**kw), "amg", tf.amg_options(jacobi_weight=2 / 3, hierarchy_type="f32"), ctx=ctx)
    s.setup(to_device(m))
    s.set_graph_mode(mode)
    return s


# guesses that leave no iteration to several; limits around the first ones
@pytest.mark.parametrize("kind", ["Cg", "BiCgStab"])
@pytest.mark.parametrize("interval", [1, 2, 5, 50])
def test_few_iterations(ctx, kind, interval):
    m = P.heat3d(14, seed=21)
    n = len(m[0]) - 1
    b = torch.tensor(P.rhs_uniform(n, 22), device="cuda")
    exact = torch.zeros_like(b)
    solver(ctx, kind, m, relative_tolerance=1e-12).apply(b, exact)
    error = torch.tensor(P.rhs_uniform(n, 23), device="cuda") * float(exact.abs().mean())
    seen = set()
    for limit in (1, 2, 3, 7, 8, 200):
        runs = [solver(ctx, kind, m, mode, max_iterations=limit, residual_refresh_interval=interval) for mode in (1, 0)]
        for size in (0.0, 1e-9, 1e-8, 1e-7, 1e-6, 1e-4, 1e-2, 1.0):
            out = []
            for s in runs:
                x = exact + size * error
                out.append((s.apply(b, x), x))
            assert out[0][0] == out[1][0], (limit, size)
            assert torch.equal(out[0][1], out[1][1]), (limit, size)
            seen.add(out[0][0]["iterations"])
    assert {0, 1, 2, 3} <= seen and max(seen) > 7, seen


def test_one_iteration_costs_no_round(ctx):
    m = P.heat3d(30, seed=24)
    n = len(m[0]) - 1
    b = torch.tensor(P.rhs_uniform(n, 25), device="cuda")

    exact = torch.zeros_like(b)
    solver(ctx, "Cg", m, relative_tolerance=1e-12).apply(b, exact)
    error = torch.tensor(P.rhs_uniform(n, 26), device="cuda") * float(exact.abs().mean())
    s = solver(ctx, "Cg", m)

    def gpu_ms(size):
        times = []
        for _ in range(9):
            x = exact + size * error
            iterations = s.apply(b, x)["iterations"]
            times.append(s.last_apply_ms)
        return iterations, min(times)

    none, many = gpu_ms(0.0), gpu_ms(1e3)
    assert none[0] == 0 and many[0] >= 20
    per_iteration = (many[1] - none[1]) / many[0]
    few = [t for t in (gpu_ms(10.0 ** -k) for k in range(5, 12)) if t[0] in (1, 2)]
    assert few
    for iterations, ms in few:
        assert ms - none[1] < (iterations + 1.5) * per_iteration, (iterations, ms, none, many)
