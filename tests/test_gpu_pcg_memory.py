"""A PCG solve at each of its device reservations failing: it ends with the
usual error, or, where only a re-laid copy of a matrix was to be made, goes on
without it to the same answer."""
import numpy as np
import pytest
from scipy import sparse

from oracle import pyoracle
from parallellocallyoptimalapproximatesparsematrixinverses_b200 import _lib, backward_error, problems

pytestmark = pytest.mark.gpu


# rows in shared memory, one chunk a cluster; and rows read from the matrices
@pytest.mark.parametrize("grid", [70, 331])
def test_solves_without_room_for_the_copies(require_gpu, grid):
    a = sparse.csr_matrix(problems.diffusion_2d(grid, 1.0, 4))
    a.sort_indices()
    m = sparse.csr_matrix(sparse.diags(1.0 / a.diagonal()))
    b = a @ np.random.default_rng(1).standard_normal(a.shape[0])
    want, want_status = pyoracle.pcg(a, m, b, 30, 1e-12, refresh_period=7, order=pyoracle.ORDER_DEVICE)
    lib = _lib.load()
    failed = []
    for after in range(40):
        lib.spai_inject_allocation_failure(after)
        try:
            hist, status = backward_error.pcg(a.data, a.indices, a.indptr, m.data, m.indices, m.indptr, b, 30, 1, 1e-12,
                                              refresh_period=7)
        except RuntimeError as error:
            assert "injected allocation failure" in str(error)
            failed.append(after)
        else:
            assert status == want_status
            assert np.array_equal(hist.view(np.int64), want.view(np.int64))
        finally:
            lib.spai_inject_allocation_failure(-1)
    # the copies are two arrays each for A and M; a later reservation still fails
    survived = [k for k in range(max(failed)) if k not in failed]
    assert len(survived) == 4
