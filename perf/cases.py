"""The calls whose speed matters to a user of this framework, as measurable cases.

A case is a dict of plain values.  `listed()` names twelve, `draw(rng)` gives
more of the same kinds and ranges.  `prepare(case, seed)` makes what a user's
program has in hand before the call (matrices, sessions, tensors), `run(state)`
is one pass through the public entry points, `exact(case, seed)` the same
outputs in 64-bit numpy where they have such a value, and `work(case)` the
bytes and operations that a pass cannot do without.

Kinds:

* mr, lomr      a resident problem (Session), per-column top-k, FP64 or mixed
                storage: building the preconditioner, the framework's main path.
* dropin        `global_spai.cg/mr/lomr` on host matrices with only the
                reference's arguments: the global budget and the reference's
                summation order over num_threads column batches.
* inner_outer   the Inner-Outer family on banded matrices with long couplings.
* batch         many small independent systems in one call.
* pcg           PCG on a resident problem with the M just built.
* pcg_grad      the differentiable solve, forward and backward, on GPU tensors.
* residual_grad ||I - A M||_F^2 and both gradients on GPU tensors.
"""
import numpy as np
import torch

from parallellocallyoptimalapproximatesparsematrixinverses_b200 import Session, adjoint, global_spai, problems


def listed():
    return [
        # the benchmark operator: 64^3 log-normal diffusion, 30 iterations, 16 entries per column, FP32 storage
        dict(name="mr_64cubed_mixed", kind="mr", grid=64, dim=3, precision="mixed", topk=16, iterations=30),
        # the same path in FP64 at an odd size and a smaller cap
        dict(name="mr_47cubed_fp64", kind="mr", grid=47, dim=3, precision="fp64", topk=12, iterations=15),
        # the small 5-point problem of the reference's CPU runs: launches and latency
        dict(name="mr_64squared_fp64", kind="mr", grid=64, dim=2, precision="fp64", topk=10, iterations=20),
        # LOMR, the method with the most products and unions per iteration
        dict(name="lomr_40cubed_mixed", kind="lomr", grid=40, dim=3, precision="mixed", topk=16, iterations=12),
        # a script of the reference switched over unchanged: default thread count, so one column batch
        dict(name="dropin_cg_1thread", kind="dropin", method="cg", grid=64, dim=2, iterations=12, per_column=24, threads=1),
        # the same with the reference's many-thread setting, in three dimensions
        dict(name="dropin_mr_64threads", kind="dropin", method="mr", grid=22, dim=3, iterations=10, per_column=40,
             threads=64),
        # Inner-Outer on a band with random couplings: wide columns, no stencil
        dict(name="inner_outer_banded", kind="inner_outer", method="lomr", n=4096, precision="mixed", topk=12,
             iterations=6),
        # many user problems at once
        dict(name="batch_24_mixed", kind="batch", count=24, n_max=16000, precision="mixed", topk=10, iterations=15),
        # evaluating M: PCG to 1e-8 on the benchmark operator
        dict(name="pcg_64cubed", kind="pcg", grid=64, dim=3, precision="mixed", topk=16, iterations=4),
        # learning through the solve: a small system, latency bound
        dict(name="pcg_grad_63squared", kind="pcg_grad", grid=63, dim=2),
        # and a large one
        dict(name="pcg_grad_300squared", kind="pcg_grad", grid=300, dim=2),
        # learning M or A against the residual objective
        dict(name="residual_grad_47cubed", kind="residual_grad", grid=47, dim=3),
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def _grid(rng, dim, lo, hi):
    """A grid edge for about lo..hi unknowns."""
    return max(3, int(round(_between(rng, lo, hi) ** (1.0 / dim))))


def draw(rng):
    kind = rng.choice(["mr", "mr", "lomr", "dropin", "dropin", "inner_outer", "batch", "pcg", "pcg_grad",
                       "residual_grad"])
    dim = rng.choice([2, 3])
    precision = rng.choice(["mixed", "fp64"])
    if kind in ("mr", "lomr"):
        return dict(kind=kind, grid=_grid(rng, dim, 4000, 200000 if kind == "mr" else 64000), dim=dim,
                    precision=precision, topk=rng.randint(8, 16), iterations=rng.randint(8, 20))
    if kind == "dropin":
        method = rng.choice(["cg", "mr", "lomr"])
        return dict(kind=kind, method=method, grid=_grid(rng, dim, 1000, 8000), dim=dim,
                    iterations=rng.randint(4, 8), per_column=rng.randint(10, 30), threads=rng.choice([1, 7, 16, 64]))
    if kind == "inner_outer":
        return dict(kind=kind, method=rng.choice(["mr", "lomr"]), n=_between(rng, 1000, 4096), precision=precision,
                    topk=rng.randint(6, 12), iterations=rng.randint(3, 6))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 32), n_max=_between(rng, 2000, 16000), precision=precision,
                    topk=rng.randint(6, 12), iterations=rng.randint(5, 15))
    if kind == "pcg":
        return dict(kind=kind, grid=_grid(rng, dim, 4000, 200000), dim=dim, precision=precision,
                    topk=rng.randint(8, 16), iterations=rng.randint(2, 6))
    return dict(kind=kind, grid=_grid(rng, dim, 4000, 90000), dim=dim)


# ---------------------------------------------------------------------------
# inputs
def _operator(case, seed):
    make = problems.diffusion_2d if case["dim"] == 2 else problems.diffusion_3d
    return make(case["grid"], 1.0, seed)


def _rows(matrix):
    """A symmetric canonical CSC matrix as CSR arrays: the same arrays."""
    return (np.ascontiguousarray(matrix.data, np.float64), np.ascontiguousarray(matrix.indices, np.int64),
            np.ascontiguousarray(matrix.indptr, np.int64))


def _neumann(a):
    """(I + N + N^2) D^-1 with N = I - D^-1 A: symmetric positive definite for
    a diagonally dominant A, and its own transpose up to rounding (the lower
    triangle is mirrored, so exactly)."""
    d = 1.0 / a.diagonal()
    scaled = a.copy()
    scaled.data = scaled.data * d[scaled.indices]
    b = scaled.copy()
    b.data = -b.data
    b.setdiag(1.0 + b.diagonal())          # N
    two = (b @ b + b).tocsc()
    two.setdiag(two.diagonal() + 1.0)      # I + N + N^2
    two.data = two.data * np.repeat(d, np.diff(two.indptr))
    m = ((two + two.T) * 0.5).tocsc()
    m.sum_duplicates()
    m.sort_indices()
    return m


def _batch(case, seed):
    """2-D and 3-D systems of 1000..n_max unknowns (their sizes are the case's, their coefficients the seed's)."""
    sizes = np.random.default_rng(case["count"] * 100003 + case["n_max"])
    systems = []
    for b in range(case["count"]):
        dim = int(sizes.integers(2, 4))
        n = float(np.exp(sizes.uniform(np.log(1000), np.log(case["n_max"]))))
        make = problems.diffusion_2d if dim == 2 else problems.diffusion_3d
        systems.append(make(int(round(n ** (1.0 / dim))), 0.5, 1000 * seed + b))
    return systems


def _cuda(values):
    return torch.from_numpy(np.array(values, dtype=np.float64)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed + 1)
    if kind in ("mr", "lomr", "pcg"):
        a = _operator(case, seed)
        n = a.shape[0]
        session = Session("global_spai", "lomr" if kind == "lomr" else "mr", a, M0=problems.diagonal_inverse(a),
                          max_iterations=case["iterations"], tolerance=1e-8, max_density=case["topk"] / n,
                          precision=case["precision"], topk_per_column=case["topk"])
        if kind == "pcg":
            session.run()
            session.set_rhs(problems.solution_rhs(a, seed)[0])
        return dict(kind=kind, session=session, precision=case["precision"])
    if kind == "dropin":
        a = _operator(case, seed)
        n = a.shape[0]
        return dict(kind=kind, method=getattr(global_spai, case["method"]), a=a, m0=problems.diagonal_inverse(a),
                    options=dict(max_iterations=case["iterations"], tolerance=1e-9,
                                 max_density=min(1.0, case["per_column"] / n), num_threads=case["threads"]))
    if kind == "inner_outer":
        a = problems.random_banded_spd(case["n"], 4, 2, seed)
        session = Session("inner_outer", case["method"], a, M0=problems.diagonal_inverse(a),
                          max_iterations=case["iterations"], tolerance=1e-9, max_density=case["topk"] / case["n"],
                          precision=case["precision"], topk_per_column=case["topk"], inner_iterations=2)
        return dict(kind=kind, session=session)
    if kind == "batch":
        systems = _batch(case, seed)
        return dict(kind=kind, systems=systems, starts=[problems.diagonal_inverse(a) for a in systems],
                    options=dict(max_iterations=case["iterations"], tolerance=1e-8,
                                 max_density=0.5, topk_per_column=case["topk"], precision=case["precision"]))
    a = _operator(case, seed)
    n = a.shape[0]
    m = _neumann(a)
    if kind == "pcg_grad":
        values, indices, offsets = _rows(a)
        mv, mi, mo = _rows(m)
        return dict(kind=kind, a=_cuda(values).requires_grad_(), b=_cuda(rng.standard_normal(n)).requires_grad_(),
                    upstream=_cuda(rng.standard_normal(n)), indices=indices, offsets=offsets, m=(mv, mi, mo))
    return dict(kind=kind, a=_cuda(a.data).requires_grad_(), m=_cuda(m.data).requires_grad_(),
                a_pattern=(np.asarray(a.indptr, np.int64), np.asarray(a.indices, np.int64)),
                m_pattern=(np.asarray(m.indptr, np.int64), np.asarray(m.indices, np.int64)))


# ---------------------------------------------------------------------------
# one pass
def _history(history):
    return [history["residual_norm"], history["density_m"], history["density_direction"]]


def run(state):
    kind = state["kind"]
    if kind in ("mr", "lomr", "inner_outer"):
        session = state["session"]
        session.run()
        m = session.result_torch()
        return dict(ptr=m.ccol_indices(), idx=m.row_indices(), val=m.values(), history=_history(session.history()))
    if kind == "dropin":
        r = state["method"](state["a"], M0=state["m0"], **state["options"])
        return dict(ptr=r.M.indptr, idx=r.M.indices, val=r.M.data, history=_history(r.history))
    if kind == "batch":
        results = global_spai.mr_batched(state["systems"], M0s=state["starts"], **state["options"])
        # one array per kind of output: the systems' results one after another
        return dict(ptr=np.concatenate([r.M.indptr for r in results]), idx=np.concatenate([r.M.indices for r in results]),
                    val=np.concatenate([r.M.data for r in results]),
                    history=[np.concatenate(column) for column in zip(*(_history(r.history) for r in results))])
    if kind == "pcg":
        history, status, x = state["session"].pcg(3000, 1e-8, refresh_period=50, m_precision=state["precision"],
                                                  return_x=True, symmetric_part=True)
        padded = np.zeros(3000)  # the number of iterations depends on the system
        padded[:history.size] = history
        return dict(history=padded, status=status, x=x)
    if kind == "pcg_grad":
        x = adjoint.pcg_solve(state["a"], state["b"], state["indices"], state["offsets"], *state["m"],
                              max_iterations=3000, tolerance=1e-9)
        grad_a, grad_b = torch.autograd.grad(x, (state["a"], state["b"]), state["upstream"])
        return dict(x=x.detach(), grad_a=grad_a, grad_b=grad_b)
    loss = adjoint.residual_objective(state["a"], state["m"], state["a_pattern"], state["m_pattern"])
    grad_a, grad_m = torch.autograd.grad(loss, (state["a"], state["m"]))
    return dict(loss=loss.detach(), grad_a=grad_a, grad_m=grad_m)


# ---------------------------------------------------------------------------
# the same outputs in plain 64-bit numpy
def _canonical(m):
    m = m.tocsc()
    m.sum_duplicates()
    m.sort_indices()
    return m


def _columns(m):
    return np.repeat(np.arange(m.shape[1]), np.diff(m.indptr))


def _select(m, keep):
    out = m.copy()
    out.data = np.where(keep, m.data, 0.0)
    out.eliminate_zeros()
    return out


def _top(m, cols, k, protect):
    """True for the k largest (|v|, row) of every column; with `protect` the diagonal comes first."""
    diagonal = (m.indices == cols) & protect
    order = np.lexsort((m.indices, np.abs(m.data), diagonal, cols))
    rank = np.empty(order.size, dtype=np.int64)
    rank[order] = np.arange(order.size) - m.indptr[:-1][cols[order]]
    return rank >= np.diff(m.indptr)[cols] - k


def _plain_drop(m, topk):
    s = _canonical((m + m.T) * 0.5)
    cols = _columns(s)
    norm = np.sqrt(np.bincount(cols, s.data ** 2, minlength=s.shape[1]))
    s = _select(s, (s.indices == cols) | (np.abs(s.data) >= np.finfo(np.float64).eps * norm[cols]))
    return _select(s, _top(s, _columns(s), topk, True))


def _scaled_rows(m, d):
    out = m.copy()
    out.data = out.data * d[out.indices]
    return out


def _dot(x, y):
    return float(x.multiply(y).sum())


def _plain_build(a, method, topk, iterations, tolerance):
    """Global MR / LOMR with per-column top-k on scipy matrices in FP64."""
    n = a.shape[0]
    d = 1.0 / a.diagonal()
    m = problems.diagonal_inverse(a).tocsc()
    identity = m.copy()
    identity.data = np.ones(n)
    m = _plain_drop(m, topk)
    r = _canonical(identity - a @ m)
    z = _scaled_rows(r, d)
    p = None
    history = [[np.sqrt(_dot(r, r)), m.nnz / n / n, (z.nnz if method == "mr" else 0) / n / n]]
    for i in range(1, iterations + 1):
        az = _canonical(a @ z)
        paz = _scaled_rows(az, d)
        if method == "mr":
            alpha = _dot(z, paz) / _dot(paz, paz)
            direction = z
            m = m + z * alpha
        else:
            gamma = 0.0
            if p is None:
                delta = _dot(z, az) / _dot(az, paz)
                p = z * 0.0
                gamma = 1.0
            else:
                ap = _canonical(a @ p)
                pap = _scaled_rows(ap, d)
                cross = _dot(az, pap)
                delta, gamma = np.linalg.solve([[_dot(az, paz), cross], [cross, _dot(ap, pap)]],
                                               [_dot(z, az), _dot(z, ap)])
            m = m + z * delta + p * gamma
            p = _canonical(z + p * (gamma / delta))
            p.eliminate_zeros()
            norm = np.sqrt(_dot(p, p))
            p = _select(p, np.abs(p.data) > np.finfo(np.float64).eps * norm)
            p = _select(p, _top(p, _columns(p), topk, False))
            direction = p
        m = _plain_drop(_canonical(m), topk)
        r = _canonical(identity - a @ m)
        r.eliminate_zeros()
        history.append([np.sqrt(_dot(r, r)), m.nnz / n / n, direction.nnz / n / n])
        if history[-1][0] < tolerance:
            break
        z = _scaled_rows(r, d)
    return m, [np.array(column) for column in zip(*history)]


def _plain_pcg(a, m, b, max_iterations, tolerance):
    x = np.zeros_like(b)
    r = b.copy()
    z = m @ r
    p = z.copy()
    rz = float(r @ z)
    norm = float(np.linalg.norm(b))
    for _ in range(max_iterations - 1):
        ap = a @ p
        alpha = rz / float(p @ ap)
        x += alpha * p
        r -= alpha * ap
        if np.linalg.norm(r) / norm <= tolerance:
            r = b - a @ x
            if np.linalg.norm(r) / norm <= tolerance:
                break
            z = m @ r
            rz, p = float(r @ z), z.copy()
            continue
        z = m @ r
        rz, before = float(r @ z), rz
        p = z + (rz / before) * p
    return x


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed + 1)
    if kind in ("mr", "lomr"):
        n = case["grid"] ** case["dim"]
        if n * case["iterations"] * (1 if kind == "mr" else 4) > 800_000:
            return None  # scipy's products would take too long
        a = _operator(case, seed)
        m, history = _plain_build(a, kind, case["topk"], case["iterations"], 1e-8)
        # in FP32 storage another entry may win a column's last place: no entrywise value for M there
        full = case["precision"] == "fp64"
        return dict(ptr=None, idx=None, val=m.data if full else None, history=[history[0], None, None])
    if kind == "pcg_grad":
        a = _operator(case, seed)
        n = a.shape[0]
        m = _neumann(a).tocsr()
        b = rng.standard_normal(n)
        upstream = rng.standard_normal(n)
        rows = a.tocsr()
        x = _plain_pcg(rows, m, b, 3000, 1e-9)
        adj = _plain_pcg(rows, m, upstream, 3000, 1e-9)
        return dict(x=x, grad_a=-adj[_columns(a)] * x[a.indices], grad_b=adj)
    if kind == "residual_grad":
        a = _operator(case, seed)
        m = _neumann(a)
        r = (a @ m) * -1.0
        r.setdiag(r.diagonal() + 1.0)
        r = _canonical(r)

        def masked(product, mask):
            """The product's values at the mask's entries (0 where it has none)."""
            keyed = _canonical(product)
            n = keyed.shape[0]
            have = _columns(keyed).astype(np.int64) * n + keyed.indices
            want = _columns(mask).astype(np.int64) * n + mask.indices
            at = np.minimum(np.searchsorted(have, want), have.size - 1)
            return np.where(have[at] == want, keyed.data[at], 0.0)

        return dict(loss=np.float64(_dot(r, r)), grad_a=-2.0 * masked(r @ m.T, a), grad_m=-2.0 * masked(a.T @ r, m))
    # dropin: last bits move the global cut; inner_outer, batch and pcg: their M has no value of its own in 64 bits
    return None


# ---------------------------------------------------------------------------
# what a pass cannot do without
def work(case):
    """Every iteration reads A and the iterate and writes the iterate, with
    the multiply-adds of its sparse products; a solve reads A and M once per
    iteration (about the typical number of them)."""
    kind = case["kind"]
    entry = 8 if case.get("precision") == "mixed" else 12
    if kind == "batch":
        n, per_row = case["count"] * case["n_max"] // 3, 6
    elif kind == "inner_outer":
        n, per_row = case["n"], 13
    else:
        n, per_row = case["grid"] ** case["dim"], 2 * case["dim"] + 1
    if kind in ("mr", "lomr", "batch", "inner_outer", "dropin"):
        width = case.get("topk") or case["per_column"]
        products = {"mr": 2, "batch": 2, "lomr": 3, "inner_outer": 4, "dropin": 3}[kind]
        per_iteration = n * (per_row + 2 * width) * entry
        flops = 2.0 * n * per_row * width * products
        return {"bytes": float(per_iteration * case["iterations"]), "flops": float(flops * case["iterations"])}
    if kind in ("pcg", "pcg_grad"):
        width = case["topk"] if kind == "pcg" else (13 if case["dim"] == 2 else 25)
        solves = 1 if kind == "pcg" else 2
        sweeps = solves * (1.3 if case["dim"] == 3 else 2.0) * case["grid"]
        return {"bytes": float(sweeps * n * (per_row * 12 + width * entry + 64)),
                "flops": float(sweeps * n * 2 * (per_row + width + 5))}
    width = 25 if case["dim"] == 3 else 13
    return {"bytes": float(n * (per_row + width) * 12 + n * (per_row + width) * 8),
            "flops": float(2.0 * n * per_row * width * 3)}
