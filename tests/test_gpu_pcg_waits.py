"""How long the blocks of a PCG solve wait for one another: a row that one
thread walks for longer than that is waited for, and the answer is the oracle's."""
import numpy as np
import pytest
from scipy import sparse

from oracle import pyoracle
from parallellocallyoptimalapproximatesparsematrixinverses_b200 import _lib, backward_error, problems

pytestmark = pytest.mark.gpu


def arrow(n):
    """A diagonal with one full row and column."""
    hub = n // 2
    others = np.delete(np.arange(n), hub)
    rows = np.concatenate([np.arange(n), np.full(n - 1, hub), others])
    cols = np.concatenate([np.arange(n), others, np.full(n - 1, hub)])
    vals = np.concatenate([np.linspace(2.0, 4.0, n), np.full(2 * (n - 1), 1.0 / n)])
    a = sparse.csr_matrix(sparse.coo_matrix((vals, (rows, cols)), shape=(n, n)))
    a.sort_indices()
    return a


def test_long_rows_are_waited_for(require_gpu):
    n = 400_000
    a = arrow(n)
    m = sparse.csr_matrix(sparse.diags(1.0 / a.diagonal()))
    b = a @ np.random.default_rng(1).standard_normal(n)
    lib = _lib.load()
    # half a millisecond: far above an exchange, far below the walk of 400,000 entries (tens of milliseconds)
    lib.spai_inject_pcg_wait(500_000)
    try:
        hist, status = backward_error.pcg(a.data, a.indices, a.indptr, m.data, m.indices, m.indptr, b, 12, 1, 1e-10)
    finally:
        lib.spai_inject_pcg_wait(-1)
    want, want_status = pyoracle.pcg(a, m, b, 12, 1e-10, order=pyoracle.ORDER_DEVICE)
    assert status == want_status
    assert np.array_equal(hist.view(np.int64), want.view(np.int64))


def _system(n_or_grid):
    if n_or_grid < 1000:
        a = sparse.csr_matrix(problems.diffusion_2d(n_or_grid, 1.0, 4))
    else:
        n = n_or_grid
        a = sparse.diags([np.full(n - 1, -1.0), np.linspace(2.5, 4.0, n), np.full(n - 1, -1.0)], [-1, 0, 1], format="csr")
    a.sort_indices()
    return a, sparse.csr_matrix(sparse.diags(1.0 / a.diagonal()))


# one chunk a cluster, several, and more than a group of rounds between cluster barriers; with a patience of 0 any
# block that does not find the others' sums at its first look gives up, some of them a reduction after the first
@pytest.mark.parametrize("size", [90, 331, 1_400_001])
def test_a_solve_that_is_given_up_ends_with_an_error(require_gpu, size):
    a, m = _system(size)
    b = a @ np.random.default_rng(1).standard_normal(a.shape[0])
    solve = lambda: backward_error.pcg(a.data, a.indices, a.indptr, m.data, m.indices, m.indptr, b, 40, 1, 1e-12,
                                       refresh_period=7)
    lib = _lib.load()
    for _ in range(5):
        lib.spai_inject_pcg_wait(0)
        try:
            with pytest.raises(RuntimeError, match="stopped answering one another"):
                solve()
        finally:
            lib.spai_inject_pcg_wait(-1)
    hist, status = solve()  # the device and the library stay usable
    want, want_status = pyoracle.pcg(a, m, b, 40, 1e-12, refresh_period=7, order=pyoracle.ORDER_DEVICE)
    assert status == want_status
    assert np.array_equal(hist.view(np.int64), want.view(np.int64))
