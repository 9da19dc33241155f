"""How long the blocks of a PCG solve wait for one another: a row that one
thread walks for longer than that is waited for, and the answer is the oracle's."""
import numpy as np
import pytest
from scipy import sparse

from oracle import pyoracle
from parallellocallyoptimalapproximatesparsematrixinverses_b200 import _lib, backward_error

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
