"""The fused Global MR kernels on groups of adjacent columns: the same bits as
the unfused kernels, at the sizes and shapes where a group changes its way --
partial groups, windows that do not hold the rows (every column on its own,
or only some of them), more rows than a group takes, short and long rows of A,
ties at the top-k cut, and thresholds that need the exact norm."""
import numpy as np
import pytest
from scipy import sparse

from parallellocallyoptimalapproximatesparsematrixinverses_b200 import _lib, global_spai, problems
from tests.helpers import assert_same_result

pytestmark = pytest.mark.gpu


def _spd(n, offsets_of, scale=1.0, seed=0):
    """Symmetric, diagonally dominant, with the off-diagonal places (rows, cols) of offsets_of(rng)."""
    rng = np.random.default_rng(seed)
    rows, cols = offsets_of(rng)
    keep = rows != cols
    off = sparse.coo_matrix((-scale * rng.uniform(0.1, 1.0, keep.sum()), (rows[keep], cols[keep])), shape=(n, n)).tocsr()
    off = off + off.T
    a = sparse.csc_matrix(off + sparse.diags(1.05 * np.asarray(abs(off).sum(axis=1)).ravel() + 0.1))
    a.sort_indices()
    return a


def _band(n, distances, seed=0):
    def places(rng):
        r = np.concatenate([np.arange(n - d) for d in distances])
        c = np.concatenate([np.arange(n - d) + d for d in distances])
        return r, c
    return _spd(n, places, seed=seed)


def _permuted(a, seed):
    p = np.random.default_rng(seed).permutation(a.shape[0])
    a = sparse.csc_matrix(a[p][:, p])
    a.sort_indices()
    return a


CASES = {
    "n1": (lambda: sparse.csc_matrix(np.array([[2.0]])), 1),
    "n5": (lambda: problems.tridiagonal(5), 3),
    "n_odd": (lambda: problems.diffusion_2d(37, 1.0, 3), 7),
    "four_columns_a_group": (lambda: problems.diffusion_2d(101, 1.0, 3), 10),
    "rows_of_3": (lambda: problems.tridiagonal(10_001), 6),
    "rows_of_9": (lambda: _band(9_999, [1, 2, 50, 51]), 12),
    "rows_of_13": (lambda: _band(9_999, [1, 2, 3, 40, 41, 90]), 32),
    # adjacent columns share nothing, inside the window: too many rows for a group
    "scattered_rows": (lambda: _permuted(problems.diffusion_2d(60, 1.0, 1), 2), 16),
    # rows further away than any window: column by column
    "wide": (lambda: _band(70_000, [1, 30_000]), 8),
    # most rows near, a few columns outside the window
    "some_columns_outside": (lambda: _band(20_000, [1, 60, 61], seed=4), 16),
    "ties": (lambda: problems.laplacian_2d(100), 6),
    "top_1": (lambda: problems.diffusion_3d(22, 1.0, 5), 1),
    "top_32": (lambda: problems.diffusion_3d(22, 1.0, 5), 32),
    # coefficients over 30 decades: entries below eps times the column's norm
    "threshold": (lambda: problems.diffusion_2d(98, 16.0, 8), 10),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", sorted(CASES))
def test_groups_match_the_unfused_kernels(require_gpu, case, precision):
    make, topk = CASES[case]
    a = make()
    n = a.shape[0]
    kw = dict(M0=problems.diagonal_inverse(a), max_iterations=9, tolerance=0.0, max_density=max(topk, 1) / n,
              topk_per_column=topk, precision=precision, summation="device")
    lib = _lib.load()
    lib.spai_set_fused_mr(0)
    try:
        want = global_spai.mr(a, **kw)
    finally:
        lib.spai_set_fused_mr(1)
    got = global_spai.mr(a, **kw)
    assert_same_result(got, want, f"{case} {precision}")


def _star(n_hubs, leaves):
    """Hubs of `leaves` neighbours: rows of M^T longer than a small cap's slots."""
    n = n_hubs * (leaves + 1)
    hub = np.repeat(np.arange(n_hubs) * (leaves + 1), leaves)
    leaf = hub + np.tile(np.arange(1, leaves + 1), n_hubs)
    return _spd(n, lambda rng: (hub, leaf), seed=1)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("systems", ["grids", "slots_outgrown"])
def test_batched_steps_match_the_unfused_kernels(require_gpu, systems, precision):
    if systems == "grids":  # groups straddle systems of odd sizes; several stop early
        batch = [problems.diffusion_2d(m, 0.5, m) for m in (3, 17, 31)] + [problems.diffusion_3d(9, 1.0, 1),
                                                                           problems.tridiagonal(5)]
        kw = dict(max_iterations=12, tolerance=0.3, max_density=1.0, topk_per_column=7, precision=precision)
    else:  # the fused steps are given up and the rest of the batch runs unfused
        batch = [_star(9, 14), problems.diffusion_2d(12, 0.5, 2)]
        kw = dict(max_iterations=6, tolerance=0.0, max_density=1.0, topk_per_column=2, precision=precision)
    lib = _lib.load()
    lib.spai_set_fused_mr(0)
    try:
        want = global_spai.mr_batched(batch, **kw)
    finally:
        lib.spai_set_fused_mr(1)
    got = global_spai.mr_batched(batch, **kw)
    for b, (g, w) in enumerate(zip(got, want)):
        assert_same_result(g, w, f"{systems} {precision} system {b}")
