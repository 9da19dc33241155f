"""The one-kernel PCG solve against the oracle, bit for bit, at the sizes where
its split changes: one row, one 32-row slice, one chunk of the tree (4,096
rows) and one more row, several clusters, and more chunks than the clusters
hold between two cluster barriers; with rows too uneven for the sliced layout."""
import numpy as np
import pytest
from scipy import sparse

from oracle import pyoracle
from parallellocallyoptimalapproximatesparsematrixinverses_b200 import backward_error, problems

pytestmark = pytest.mark.gpu


def _tridiagonal(n):
    main = np.linspace(2.5, 4.0, n)
    off = np.full(n - 1, -1.0)
    return sparse.diags([off, main, off], [-1, 0, 1], format="csr")


def _uneven(n):
    """A few dense rows among diagonal ones: their slices stay row-compressed."""
    rng = np.random.default_rng(3)
    hubs = np.arange(0, n, 97)
    rows = np.repeat(hubs, 60)
    cols = rng.integers(0, n, rows.size)
    vals = rng.uniform(0.1, 0.5, rows.size)
    a = sparse.coo_matrix((vals, (rows, cols)), shape=(n, n)).tocsr()
    a = a + a.T
    a.setdiag(1.1 * np.asarray(abs(a).sum(axis=1)).ravel() + 1.0)
    return sparse.csr_matrix(a)


CASES = {
    "one_row": (lambda: sparse.csr_matrix(np.array([[3.0]])), 5, 0),
    "one_slice": (lambda: _tridiagonal(31), 60, 0),
    "one_chunk": (lambda: _tridiagonal(4096), 40, 7),
    "one_chunk_and_a_row": (lambda: _tridiagonal(4097), 40, 7),
    "uneven_rows": (lambda: _uneven(9001), 60, 10),
    "many_clusters": (lambda: sparse.csr_matrix(problems.diffusion_2d(331, 1.0, 4)), 50, 20),
    "two_blocks_per_sm": (lambda: sparse.csr_matrix(problems.diffusion_3d(61, 1.0, 4)), 30, 13),
    "several_groups_of_rounds": (lambda: _tridiagonal(1_400_001), 9, 4),
}


@pytest.mark.parametrize("symmetric_part", [False, True])
@pytest.mark.parametrize("case", sorted(CASES))
def test_solve_matches_the_oracle(require_gpu, case, symmetric_part):
    make, iterations, refresh = CASES[case]
    a = make()
    a.sort_indices()
    n = a.shape[0]
    d = 1.0 / a.diagonal()
    m = a.copy()  # D^-1 A D^-1-like pattern, diagonally dominant: 2 D^-1 - D^-1 A D^-1
    m.data = -m.data * d[m.indices] * np.repeat(d, np.diff(m.indptr))
    m.setdiag(m.diagonal() + 2.0 * d)
    m = sparse.csr_matrix((m + m.T) * 0.5)
    m.sort_indices()
    b = a @ np.random.default_rng(1).standard_normal(n)
    hist, status, x = backward_error.pcg(a.data, a.indices, a.indptr, m.data, m.indices, m.indptr, b, iterations, 1,
                                         1e-10, refresh_period=refresh, return_x=True, symmetric_part=symmetric_part)
    want, want_status = pyoracle.pcg(a, m, b, iterations, 1e-10, refresh_period=refresh,
                                     order=pyoracle.ORDER_DEVICE)
    assert status == want_status
    assert np.array_equal(hist.view(np.int64), want.view(np.int64))
    assert np.linalg.norm(b - a @ x) <= 1.01 * hist[-1] * np.linalg.norm(b) + 1e-12


def test_concurrent_solves_from_several_threads(require_gpu):
    from concurrent.futures import ThreadPoolExecutor
    a = sparse.csr_matrix(problems.diffusion_2d(150, 1.0, 2))
    a.sort_indices()
    m = sparse.diags(1.0 / a.diagonal(), format="csr")
    bs = [a @ np.random.default_rng(k).standard_normal(a.shape[0]) for k in range(6)]

    def solve(b):
        return backward_error.pcg(a.data, a.indices, a.indptr, m.data, m.indices, m.indptr, b, 200, 1, 1e-9)

    alone = [solve(b) for b in bs]
    with ThreadPoolExecutor(max_workers=6) as pool:
        together = list(pool.map(solve, bs))
    for (h0, s0), (h1, s1) in zip(alone, together):
        assert s0 == s1 and np.array_equal(h0.view(np.int64), h1.view(np.int64))
