"""Sums in the reference's order of several long column batches (each over
16,384 entries: eight blocks a batch), several tiles long and ending inside a
piece, against the oracle; sums that are not finite; and the reference's order
with FP32 storage."""
import numpy as np
import pytest
from scipy import sparse

from oracle import pyoracle
from parallellocallyoptimalapproximatesparsematrixinverses_b200 import global_spai, inner_outer, problems
from tests.helpers import assert_same_result

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [2, 5])
@pytest.mark.parametrize("method", ["cg", "mr"])
def test_several_long_batches_match_the_oracle(require_gpu, method, threads):
    A = problems.diffusion_2d(101, 1.0, 5)
    kw = dict(M0=problems.diagonal_inverse(A), max_iterations=4, tolerance=1e-12, max_density=14.0 / A.shape[0],
              num_threads=threads)
    got = getattr(global_spai, method)(A, **kw)
    want = pyoracle.run("global_spai", method, A, order=pyoracle.ORDER_REFERENCE, **kw)
    assert 14 * A.shape[0] // threads > 16384
    assert_same_result(got, want, f"{method} {threads} threads")


def _spoiled(value):
    a = problems.diffusion_2d(100, 1.0, 3).tolil()
    a[7, 8] = a[8, 7] = value
    return sparse.csc_matrix(a)


# one long batch (eight blocks), batches of a few thousand entries (256 threads) and of a few (32)
@pytest.mark.parametrize("threads", [1, 16, 1000])
@pytest.mark.parametrize("value", [1e200, np.inf, np.nan])
def test_sums_that_are_not_finite_match_the_oracle(require_gpu, value, threads):
    A = _spoiled(value)
    kw = dict(M0=problems.diagonal_inverse(A), max_iterations=3, tolerance=1e-12, max_density=14.0 / A.shape[0],
              num_threads=threads)
    got = global_spai.cg(A, **kw)
    want = pyoracle.run("global_spai", "cg", A, order=pyoracle.ORDER_REFERENCE, **kw)
    assert got.iterations == want.iterations
    assert np.array_equal(got.history["residual_norm"], want.history["residual_norm"], equal_nan=True)
    assert not np.isfinite(got.history["residual_norm"][0])
    assert (sparse.csc_matrix(got.M) != sparse.csc_matrix(want.M)).nnz == 0


# per-column coefficients: the spoiled columns stay, their directions' top-k is by rank
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_topk_of_columns_with_nan_matches_the_oracle(require_gpu, value):
    A = _spoiled(value)
    kw = dict(M0=problems.diagonal_inverse(A), max_iterations=3, tolerance=1e-12, max_density=4.0 / A.shape[0])
    got = inner_outer.lomr(A, topk_per_column=4, summation="device", **kw)
    want = pyoracle.run("inner_outer", "lomr", A, topk_per_column=4, order=pyoracle.ORDER_DEVICE, **kw)
    assert got.iterations == want.iterations
    gm, wm = sparse.csc_matrix(got.M), sparse.csc_matrix(want.M)
    assert np.array_equal(gm.indptr, wm.indptr) and np.array_equal(gm.indices, wm.indices)
    assert np.array_equal(gm.data, wm.data, equal_nan=True)


# The first residual's entries do not depend on the order; its sum of squares, in 64 bits, differs by at most one
# rounding per term.
@pytest.mark.parametrize("threads", [1, 16, 1000])
@pytest.mark.parametrize("method", ["cg", "mr", "lomr"])
def test_reference_order_with_fp32_storage(require_gpu, method, threads):
    A = problems.diffusion_2d(100, 1.0, 3)
    kw = dict(M0=problems.diagonal_inverse(A), max_iterations=3, tolerance=1e-12, max_density=14.0 / A.shape[0],
              precision="mixed")
    run = getattr(global_spai, method)
    ordered = run(A, num_threads=threads, summation="reference", **kw).history["residual_norm"]
    tree = run(A, summation="device", **kw).history["residual_norm"]
    assert abs(ordered[0] - tree[0]) <= A.nnz * np.finfo(np.float64).eps * tree[0]
    # later ones: the step lengths differ by such roundings, M's FP32 entries by one of theirs
    scale = np.sqrt(A.shape[0]) * np.finfo(np.float32).eps * 100
    assert ordered.size == tree.size and np.all(np.abs(ordered - tree) <= scale)
