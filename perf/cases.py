"""The calls a user of this library makes, as measurable cases.

A case names a kind of call (KINDS below), an operator, its size and the
options of the call.  The operators are the ones the repository's workloads
use, generated on the GPU from the seed: 7-point heat conduction with
log-normal conductivity, 7-point convection-diffusion with upwind convection,
the backward-Euler step of a heat problem, the 2-D 5-point Laplacian, and an
unstructured graph Laplacian with ragged rows (a mesh whose numbering follows
no grid).

  spmv      y = A x with the caller's CSR arrays
  smooth    a weighted Jacobi smoother (two sweeps) on the caller's CSR arrays
  cycle     one application of a built AMG preconditioner
  setup     an AMG preconditioner for a new operator and its first application
  solve     a whole PCG or BiCGStab solve to 1e-8 with a built solver
  batch     one time step of several systems solved together
  train     one minibatch step of the learned damping network
"""
import math

import torch

import thermofem_b200 as tf

# ---------------------------------------------------------------------------
# operators (CSR on the GPU, FP64 values, int32 indices)
# ---------------------------------------------------------------------------


def _generator(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + stream) % (1 << 62))
    return g


def _uniform(n, seed, stream):
    """n values uniform in [-1, 1]."""
    return 2 * torch.rand(n, dtype=torch.float64, device="cuda", generator=_generator(seed, stream)) - 1


def _grid(nx, ny, nz):
    i = torch.arange(nx * ny * nz, device="cuda", dtype=torch.int32)
    ix, iy, iz = i % nx, (i // nx) % ny, i // (nx * ny)
    steps = (-nx * ny, -nx, -1, 1, nx, nx * ny)
    inside = (iz > 0, iy > 0, ix > 0, ix < nx - 1, iy < ny - 1, iz < nz - 1)
    return i, ix, steps, inside


def _stencil(i, steps, inside, couplings, diagonal):
    """CSR of a stencil: entries in column order, absent neighbours left out."""
    half = len(steps) // 2
    order = [*range(half), None, *range(half, len(steps))]
    cols = torch.stack([i if k is None else i + steps[k] for k in order], 1)
    vals = torch.stack([diagonal if k is None else couplings[k] for k in order], 1)
    keep = torch.stack([torch.ones_like(inside[0]) if k is None else inside[k] for k in order], 1)
    offsets = torch.zeros(i.numel() + 1, dtype=torch.int32, device="cuda")
    offsets[1:] = keep.sum(1).cumsum(0)
    return offsets, cols[keep], vals[keep]


def _heat(nx, ny, nz, seed):
    """Harmonic-mean face coefficients of a log-normal conductivity, T = 0 on the face x = 0, insulated elsewhere."""
    i, ix, steps, inside = _grid(nx, ny, nz)
    k = torch.exp(torch.randn(i.numel(), dtype=torch.float64, device="cuda", generator=_generator(seed, 1)))
    h2 = 1.0 / nx**2
    couplings, diagonal = [], torch.where(ix == 0, 2 * k / h2, 0.0)
    for step, ok in zip(steps, inside):
        kj = k[torch.where(ok, i + step, i)]
        face = torch.where(ok, 2 * k * kj / (k + kj) / h2, 0.0)
        couplings.append(-face)
        diagonal = diagonal + face
    return _stencil(i, steps, inside, couplings, diagonal)


def _convdiff(nx, ny, nz, seed):
    """Diffusion plus upwind convection in a random direction, cell Peclet number in [1, 10], Robin on x = 0 and x = 1."""
    i, ix, steps, inside = _grid(nx, ny, nz)
    u = torch.rand(3, dtype=torch.float64, device="cuda", generator=_generator(seed, 2)).tolist()
    z, phi, peclet = 2 * u[0] - 1, 2 * math.pi * u[1], 1 + 9 * u[2]
    r, h = math.sqrt(max(0.0, 1 - z * z)), 1.0 / nx
    v = [2 * peclet / h * d for d in (r * math.cos(phi), r * math.sin(phi), z)]
    couplings, diagonal = [], torch.zeros(i.numel(), dtype=torch.float64, device="cuda")
    for k, (axis, sign) in enumerate(zip((2, 1, 0, 0, 1, 2), (-1, -1, -1, 1, 1, 1))):
        out = sign * v[axis]
        couplings.append(torch.where(inside[k], -1 / h**2 - max(-out, 0.0) / h, 0.0))
        diagonal = diagonal + torch.where(inside[k], 1 / h**2 + max(out, 0.0) / h, 0.0)
    robin = 1 / (h / 2 + 0.1) / h
    diagonal = diagonal + torch.where(ix == 0, robin, 0.0) + torch.where(ix == nx - 1, robin, 0.0)
    return _stencil(i, steps, inside, couplings, diagonal)


def _transient(n, r):
    """(1/r) I + K7 on n^3 cells with Dirichlet walls, the backward-Euler step operator."""
    i, _, steps, inside = _grid(n, n, n)
    one = torch.ones(i.numel(), dtype=torch.float64, device="cuda")
    return _stencil(i, steps, inside, [-one] * 6, (6 + 1 / r) * one)


def _laplace(nx, ny):
    """5-point Laplacian with homogeneous Dirichlet boundaries."""
    i = torch.arange(nx * ny, device="cuda", dtype=torch.int32)
    ix, iy = i % nx, i // nx
    one = torch.ones(i.numel(), dtype=torch.float64, device="cuda") * (nx + 1.0) ** 2
    return _stencil(i, (-nx, -1, 1, nx), (iy > 0, ix > 0, ix < nx - 1, iy < ny - 1), [-one] * 4, 4 * one)


def _graph(n, seed):
    """Weighted graph Laplacian plus a small mass term: 1 to 12 edges out of
    every vertex to vertices within n/64, every 16th vertex one far edge."""
    g = _generator(seed, 3)
    degree = 1 + (12 * torch.rand(n, device="cuda", generator=g) ** 3).long()
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), degree)
    reach = max(4, n // 64)
    dst = (src + torch.randint(1, reach + 1, src.shape, device="cuda", generator=g)) % n
    far = torch.arange(0, n, 16, device="cuda")
    src = torch.cat([src, far])
    dst = torch.cat([dst, torch.randint(0, n, far.shape, device="cuda", generator=g)])
    off_diagonal = src != dst
    src, dst = src[off_diagonal], dst[off_diagonal]
    edge = torch.unique(torch.minimum(src, dst) * n + torch.maximum(src, dst))
    a, b = edge // n, edge % n
    # weights are multiples of 2^-20, so that their sums are exact in any order
    w = torch.exp(torch.randn(edge.numel(), dtype=torch.float64, device="cuda", generator=g))
    w = (w * 2**20).ceil() / 2**20
    diagonal = torch.full((n,), 2.0**-4, dtype=torch.float64, device="cuda")
    diagonal.index_add_(0, a, w).index_add_(0, b, w)
    i = torch.arange(n, device="cuda")
    rows, cols = torch.cat([a, b, i]), torch.cat([b, a, i])
    order = torch.argsort(rows * n + cols)
    rows, cols, vals = rows[order], cols[order], torch.cat([-w, -w, diagonal])[order]
    offsets = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    offsets[1:] = torch.bincount(rows, minlength=n).cumsum(0)
    return offsets.int(), cols.int(), vals


def _operator(case, seed):
    """(offsets, indices, values) of the case's operator."""
    kind = case["operator"]
    if kind == "heat":
        return _heat(case["nx"], case["ny"], case["nz"], seed)
    if kind == "convdiff":
        return _convdiff(case["nx"], case["ny"], case["nz"], seed)
    if kind == "laplace":
        return _laplace(case["nx"], case["ny"])
    return _graph(case["rows"], seed)


def _rows(case):
    if case["operator"] == "graph":
        return case["rows"]
    return case["nx"] * case["ny"] * case.get("nz", 1)


def _entries(case):
    """Nonzeros (for the graph: close to what its distribution gives)."""
    if case["operator"] == "graph":
        return int(case["rows"] * 8.5)
    nx, ny, nz = case["nx"], case["ny"], case.get("nz", 1)
    n = nx * ny * nz
    return n + 2 * (n - ny * nz) + 2 * (n - nx * nz) + (2 * (n - nx * ny) if nz > 1 else 0)


_DTYPE = {"f64": torch.float64, "f32": torch.float32}
OMEGA = (0.3, 1.2)  # bounds of the network's output
_INDEX = {"i32": torch.int32, "i64": torch.int64}


def _csr(case, seed):
    offsets, indices, values = _operator(case, seed)
    index = _INDEX[case.get("index", "i32")]
    return tf.DeviceCsr(offsets.to(index), indices.to(index), values.to(_DTYPE[case["dtype"]]))


def _amg_options(case):
    return tf.amg_options(cycle=case["cycle"], hierarchy_type=case["hierarchy"], jacobi_weight=2 / 3)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the operator product of a caller's own time loop, FP64 CSR beyond the L2 cache
        {"name": "spmv_heat_f64", "kind": "spmv", "operator": "heat", "nx": 192, "ny": 192, "nz": 192,
         "dtype": "f64", "index": "i32"},
        # an unstructured mesh's operator, single precision, 64-bit indices, a row count that divides by nothing
        {"name": "spmv_graph_f32", "kind": "spmv", "operator": "graph", "rows": 300007, "dtype": "f32",
         "index": "i64"},
        # the smoother component on its own, as inside a caller's own multigrid
        {"name": "smooth_convdiff_f64", "kind": "smooth", "operator": "convdiff", "nx": 97, "ny": 96, "nz": 95,
         "dtype": "f64"},
        # the preconditioner inside a caller's own FP64 Krylov loop, FP32 hierarchy
        {"name": "vcycle_heat_mixed", "kind": "cycle", "operator": "heat", "nx": 160, "ny": 160, "nz": 160,
         "dtype": "f64", "hierarchy": "f32", "cycle": "v"},
        # the many small visits of a W-cycle, FP64 throughout
        {"name": "wcycle_convdiff_f64", "kind": "cycle", "operator": "convdiff", "nx": 80, "ny": 80, "nz": 80,
         "dtype": "f64", "hierarchy": "f64", "cycle": "w"},
        # a new operator every time (changed coefficients): what precedes the first solve
        {"name": "setup_heat_mixed", "kind": "setup", "operator": "heat", "nx": 128, "ny": 128, "nz": 128,
         "dtype": "f64", "hierarchy": "f32", "cycle": "v"},
        # the same for an unstructured mesh in FP64
        {"name": "setup_graph_f64", "kind": "setup", "operator": "graph", "rows": 60013, "dtype": "f64",
         "hierarchy": "f64", "cycle": "f"},
        # the small 2-D problem: latency of a whole solve
        {"name": "cg_laplace_small", "kind": "solve", "solver": "cg", "operator": "laplace", "nx": 128, "ny": 128,
         "dtype": "f64", "hierarchy": "f64", "cycle": "v", "host": False},
        # the headline problem: 256^3 heat conduction, FP32 hierarchy under FP64 PCG
        {"name": "cg_heat_256_mixed", "kind": "solve", "solver": "cg", "operator": "heat", "nx": 256, "ny": 256,
         "nz": 256, "dtype": "f64", "hierarchy": "f32", "cycle": "v", "host": False},
        # nonsymmetric, W-cycle, vectors in pinned host memory
        {"name": "bicgstab_convdiff", "kind": "solve", "solver": "bicgstab", "operator": "convdiff", "nx": 112,
         "ny": 112, "nz": 112, "dtype": "f64", "hierarchy": "f32", "cycle": "w", "host": True},
        # uneven transient systems advanced together
        {"name": "batch_transient", "kind": "batch", "systems": 12, "side_min": 16, "side_max": 64, "layout": 1004},
        # the damping network's minibatch step
        {"name": "train_damping", "kind": "train", "rows": 32768},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    m = _log_int(rng, lo, hi)
    return {"nx": m, "ny": max(4, m + rng.randint(-3, 3)), "nz": max(4, m + rng.randint(-3, 3))}


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "smooth", "cycle", "cycle", "setup", "setup", "solve", "solve", "batch", "train"])
    if kind == "batch":
        lo = rng.randint(16, 32)
        return {"kind": "batch", "systems": rng.randint(2, 16), "side_min": lo, "side_max": rng.randint(lo + 8, 72),
                "layout": rng.randint(1, 1 << 20)}
    if kind == "train":
        return {"kind": "train", "rows": _log_int(rng, 2048, 131072)}
    case = {"kind": kind, "operator": rng.choice(["heat", "heat", "convdiff", "laplace", "graph"])}
    cycle = rng.choice(["v", "v", "w", "f"])
    top = {"spmv": 224, "smooth": 192, "cycle": 192, "setup": 144, "solve": 176}[kind]
    if kind == "solve" and case["operator"] == "graph":
        case["operator"] = "heat"
    if case["operator"] == "graph":
        case["rows"] = _log_int(rng, 2000, 1500000 if kind in ("spmv", "smooth") else 300000)
    elif case["operator"] == "laplace":
        m = _log_int(rng, 48, 1400 if kind in ("spmv", "smooth") else 700)
        case.update(nx=m, ny=m + rng.randint(-5, 5))
    else:
        if kind == "solve" and (case["operator"] == "convdiff" or cycle != "v"):
            top = 104
        case.update(_box(rng, 14, top))
    if kind in ("spmv", "smooth"):
        case["dtype"] = rng.choice(["f64", "f64", "f32"])
        if kind == "spmv":
            case["index"] = rng.choice(["i32", "i32", "i64"])
        return case
    case.update(dtype="f64", hierarchy=rng.choice(["f32", "f32", "f64", "f32v"]), cycle=cycle)
    if kind == "solve":
        # PCG on the symmetric operators, BiCGStab on the other
        case["solver"] = "bicgstab" if case["operator"] == "convdiff" else "cg"
        case["host"] = rng.random() < 0.3
        if case["operator"] == "convdiff":
            case["hierarchy"] = rng.choice(["f32", "f64"])
    return case


# ---------------------------------------------------------------------------
# state and pass
# ---------------------------------------------------------------------------


def _batch_systems(case):
    """(side, r) of every system: side uniform in the range, r = dt k / h^2 in [0.1, 10]; the program's fixed set of parts."""
    g = torch.Generator()
    g.manual_seed(case["layout"])
    u = torch.rand(case["systems"], 2, generator=g, dtype=torch.float64).tolist()
    span = case["side_max"] - case["side_min"] + 1
    return [(case["side_min"] + min(int(a * span), span - 1), 0.1 + 9.9 * b) for a, b in u]


def _train_data(case, seed):
    """Row features and targets as the training set has them (four features per row, targets among the candidates)."""
    n = case["rows"]
    g = _generator(seed, 5)
    x = torch.empty((n, 4), dtype=torch.float32, device="cuda")
    x[:, 0] = 1.2 * torch.randn(n, device="cuda", generator=g)
    x[:, 1] = 1 - 0.3 * torch.rand(n, device="cuda", generator=g) ** 4
    x[:, 2] = torch.randint(4, 40, (n,), device="cuda", generator=g) / 8
    x[:, 3] = torch.randint(0, 8, (n,), device="cuda", generator=g) / 10
    candidates = torch.tensor([0.5, 0.6, 0.7, 0.8, 0.9, 1.0], device="cuda")
    return x, candidates[torch.randint(0, 6, (n,), device="cuda", generator=g)]


def _train_weights(seed):
    """Initial FP32 weights: Glorot-uniform layers, an output near 2/3."""
    g = torch.Generator()
    g.manual_seed(int(seed) % (1 << 62))
    p = torch.zeros(193)
    p[:128] = math.sqrt(6 / 36) * (2 * torch.rand(128, generator=g) - 1)
    p[160:192] = math.sqrt(6 / 33) * (2 * torch.rand(32, generator=g) - 1)
    p[192] = -0.37
    return p


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "train":
        state["features"], state["targets"] = _train_data(case, seed)
        state["model"] = tf.Mlp(omega_min=OMEGA[0], omega_max=OMEGA[1], params=_train_weights(seed).numpy())
        return state
    if kind == "batch":
        solvers, start, rhs_of = [], [], []
        for k, (side, r) in enumerate(_batch_systems(case)):
            a = tf.DeviceCsr(*_transient(side, r))
            s = tf.Cg(tf.solver_options(), "amg", tf.amg_options(hierarchy_type="f32"))
            s.setup(a)
            solvers.append(s)
            t0 = (_uniform(a.rows, seed, 100 + k) + 1) / 2
            start.append(t0)
            rhs_of.append(t0 / r)
        sizes = [t.numel() for t in start]
        state["batch"] = tf.Batch(solvers)
        state["start"], state["rhs"] = torch.cat(start), torch.cat(rhs_of).split(sizes)
        state["x"] = torch.empty_like(state["start"])
        state["views"] = state["x"].split(sizes)
        return state
    a = _csr(case, seed)
    state["a"] = a
    dtype = _DTYPE[case["dtype"]]
    b = _uniform(a.rows, seed, 10).to(dtype)
    if kind == "spmv":
        state["x"], state["y"] = b, torch.empty_like(b)
    elif kind == "smooth":
        state["b"], state["guess"] = b, _uniform(a.rows, seed, 11).to(dtype)
        state["x"] = torch.empty_like(b)
        state["smoother"] = tf.Jacobi(sweeps=2, dtype=dtype)
        state["smoother"].setup(a)
    elif kind == "cycle":
        state["b"], state["x"] = b, torch.empty_like(b)
        state["amg"] = tf.Amg(_amg_options(case), dtype=dtype)
        state["amg"].setup(a)
    elif kind == "setup":
        state["b"] = b
    else:
        cls = tf.Cg if case["solver"] == "cg" else tf.BiCgStab
        state["solver"] = cls(tf.solver_options(), "amg", _amg_options(case))
        state["solver"].setup(a)
        if case["host"]:
            state["b"] = torch.empty(a.rows, dtype=dtype, pin_memory=True).copy_(b)
            state["x"] = torch.empty(a.rows, dtype=dtype, pin_memory=True)
        else:
            state["b"], state["x"] = b, torch.empty_like(b)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "spmv":
        return tf.spmv(state["a"], state["x"], state["y"])
    if kind == "smooth":
        state["x"].copy_(state["guess"])
        return state["smoother"].apply(state["b"], state["x"])
    if kind == "cycle":
        return state["amg"].apply(state["b"], state["x"])
    if kind == "setup":
        amg = tf.Amg(_amg_options(case), dtype=_DTYPE[case["dtype"]])
        amg.setup(state["a"])
        levels = amg.level_statistics()
        return {"x": amg.apply(state["b"]), "rows": [v["rows"] for v in levels], "nonzeros": [v["nonzeros"] for v in levels]}
    if kind == "solve":
        state["x"].zero_()
        state["solver"].apply(state["b"], state["x"])
        return state["x"]
    if kind == "batch":
        state["x"].copy_(state["start"])
        state["batch"].apply(state["rhs"], state["views"])
        return state["x"]
    loss = state["model"].backward(state["features"], state["targets"])
    gradient = state["model"].gradient()
    state["model"].sgd(0.5, 0.9)
    return {"loss": loss, "gradient": gradient, "params": state["model"].params()}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def _iterations(case):
    """Iterations such a solve takes (measured on the listed sizes)."""
    m = case["nx"]
    return math.ceil({"laplace": 4.2, "heat": 8.7, "convdiff": 3.4}[case["operator"]] * math.sqrt(m))


def _cycle_bytes(n, nnz, value):
    """One cycle: the operator three times (residual, sweep after the coarse
    correction, the coarser levels' operators together about once more),
    about eight vectors."""
    return 3 * nnz * (value + 4) + 8 * n * value


def work(case):
    kind = case["kind"]
    if kind == "train":
        return {"bytes": case["rows"] * 20, "flops": case["rows"] * 32 * 4 * 6}
    if kind == "batch":
        total = 0
        for side, _ in _batch_systems(case):
            n = side**3
            nnz = 7 * n - 6 * side * side
            total += 8 * (nnz * 12 + 10 * n * 8 + _cycle_bytes(n, nnz, 4))
        return {"bytes": total, "flops": total / 4}
    n, nnz = _rows(case), _entries(case)
    value = 8 if case["dtype"] == "f64" else 4
    index = 8 if case.get("index") == "i64" else 4
    if kind == "spmv":
        return {"bytes": nnz * (value + index) + n * (index + 2 * value), "flops": 2 * nnz}
    if kind == "smooth":
        return {"bytes": 2 * (nnz * (value + 4) + n * (4 + 4 * value)), "flops": 4 * nnz}
    cycle = _cycle_bytes(n, nnz, 8 if case["hierarchy"] == "f64" else 4)
    if kind == "cycle":
        return {"bytes": cycle, "flops": cycle / 4}
    if kind == "setup":
        # the operator read and every level's operator (about as much again) written, the graph and product in between
        return {"bytes": 4 * nnz * 12 + cycle, "flops": 4 * nnz}
    applications = 1 if case["solver"] == "cg" else 2
    total = _iterations(case) * applications * (nnz * 12 + 10 * n * 8 + cycle)
    return {"bytes": total, "flops": total / 4}


# ---------------------------------------------------------------------------
# the same results in 64 bits, by plain torch
# ---------------------------------------------------------------------------


def _sparse(offsets, indices, values):
    n = offsets.numel() - 1
    return torch.sparse_csr_tensor(offsets.long(), indices.long(), values, size=(n, n))


def _diagonal(offsets, indices, values):
    rows = torch.repeat_interleave(torch.arange(offsets.numel() - 1, device="cuda"), offsets.diff().long())
    on = indices == rows
    d = torch.zeros(offsets.numel() - 1, dtype=torch.float64, device="cuda")
    d[rows[on]] = values[on]
    return d


def _cg64(a, d, b, limit=6000):
    """Jacobi-preconditioned CG to the end of FP64; None when it gets stuck."""
    x = torch.zeros_like(b)
    r, z = b.clone(), b / d
    p, rho, norm = z.clone(), torch.dot(b, z), torch.linalg.norm(b)
    for it in range(limit):
        q = a @ p
        alpha = rho / torch.dot(p, q)
        x += alpha * p
        r -= alpha * q
        if it % 20 == 0 and float(torch.linalg.norm(r) / norm) < 1e-13:
            return x
        z = r / d
        new = torch.dot(r, z)
        p = z + (new / rho) * p
        rho = new
    return None


def _bicgstab64(a, d, b, limit=3000):
    """Jacobi-preconditioned BiCGStab, restarted from the true residual until that is 1e-12; None when it gets stuck."""
    x, norm = torch.zeros_like(b), torch.linalg.norm(b)
    done = 0
    while done < limit:
        r = b - a @ x
        if float(torch.linalg.norm(r) / norm) < 1e-12:
            return x
        shadow, p, rho = r.clone(), r.clone(), torch.dot(r, r)
        goal = max(1e-13 * float(norm), 1e-6 * float(torch.linalg.norm(r)))
        for it in range(600):
            done += 1
            ph = p / d
            v = a @ ph
            alpha = rho / torch.dot(shadow, v)
            s = r - alpha * v
            sh = s / d
            t = a @ sh
            omega = torch.dot(t, s) / torch.dot(t, t)
            x = x + alpha * ph + omega * sh
            r = s - omega * t
            if it % 10 == 0 and not float(torch.linalg.norm(r)) > goal:
                break
            new = torch.dot(shadow, r)
            p = r + (new / rho) * (alpha / omega) * (p - omega * v)
            rho = new
        if not bool(torch.isfinite(x).all()):
            return None
    return None


def _exact_train(case, seed):
    """The loss, its summed gradient and the first SGD step in 64 bits from the network's initial FP32 weights."""
    initial = _train_weights(seed)
    p = initial.to(torch.bfloat16).double()
    x, t = _train_data(case, seed)
    x, t = x.double().cpu(), t.double().cpu()
    w1, b1, w2, b2 = p[:128].view(32, 4), p[128:160], p[160:192], p[192]
    lo, hi = torch.tensor(OMEGA, dtype=torch.float32).double()
    a = x @ w1.T + b1
    h = a.clamp(min=0)
    s = 1 / (1 + torch.exp(-(h @ w2 + b2)))
    e = lo + (hi - lo) * s - t
    dz = 2 * e * (hi - lo) * s * (1 - s)
    dh = torch.where(a > 0, dz[:, None] * w2[None, :], 0.0)
    g = torch.cat([(dh.T @ x).reshape(-1), dh.sum(0), (dz[:, None] * h).sum(0), dz.sum()[None]])
    mean = g / case["rows"]
    return {"loss": float((e * e).mean()), "gradient": g, "params": initial.double() - 0.5 * mean}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind in ("cycle", "setup"):
        return None  # what a cycle gives depends on the aggregates, which only the hierarchy itself defines
    if kind == "batch":
        out = []
        for k, (side, r) in enumerate(_batch_systems(case)):
            op = _transient(side, r)
            out.append(_cg64(_sparse(*op), _diagonal(*op), (_uniform(side**3, seed, 100 + k) + 1) / 2 / r))
        return torch.cat(out)
    dtype = _DTYPE[case["dtype"]]
    offsets, indices, values = _operator(case, seed)
    values = values.to(dtype).double()
    a = _sparse(offsets, indices, values)
    b = _uniform(offsets.numel() - 1, seed, 10).to(dtype).double()
    if kind == "spmv":
        return a @ b
    d = _diagonal(offsets, indices, values)
    if kind == "smooth":
        x = _uniform(b.numel(), seed, 11).to(dtype).double()
        for _ in range(2):
            x = x + 2 / 3 * (b - a @ x) / d
        return x
    return _cg64(a, d, b) if case["solver"] == "cg" else _bicgstab64(a, d, b)
