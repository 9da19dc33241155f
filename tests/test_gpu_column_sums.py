"""Per-column sums and the per-column top-k of a direction against the oracle,
bit for bit: column counts that do not fill a warp's four, columns from one
entry to about a thousand, equal and different patterns, ties at the cut (the
Laplacian's repeated magnitudes), caps of one entry and of more than a warp."""
import numpy as np
import pytest
from scipy import sparse

from oracle import pyoracle
from parallellocallyoptimalapproximatesparsematrixinverses_b200 import global_spai, inner_outer, problems
from tests.helpers import assert_same_result

pytestmark = pytest.mark.gpu



def arrow(n):
    """Columns of two entries beside one of n: staged rows up to 256, longer ones read in place."""
    a = sparse.lil_matrix((n, n))
    a[-1, :] = a[:, -1] = -0.25 + np.arange(n) / (16.0 * n)
    a.setdiag(n)
    return sparse.csc_matrix(a)


OPERATORS = {
    "arrow_256": lambda: arrow(256),
    "arrow_257": lambda: arrow(257),
    "tridiagonal_6": lambda: problems.tridiagonal(6),
    "laplacian_33": lambda: problems.laplacian_2d(33),
    "diffusion_3d_9": lambda: problems.diffusion_3d(9, 1.0, 2),
    "banded_1001": lambda: problems.random_banded_spd(1001, 4, 3, seed=5),
}


@pytest.mark.parametrize("topk", [1, 7, 40])
@pytest.mark.parametrize("operator", sorted(OPERATORS))
@pytest.mark.parametrize("family,name", [("global_spai", "cg"), ("global_spai", "lomr"), ("inner_outer", "lomr")])
def test_sums_and_topk_match_the_oracle(require_gpu, family, name, operator, topk):
    A = OPERATORS[operator]()
    kw = dict(M0=problems.diagonal_inverse(A), max_iterations=4, tolerance=0.0,
              max_density=min(1.0, max(topk, 2) / A.shape[0]))
    method = getattr({"global_spai": global_spai, "inner_outer": inner_outer}[family], name)
    got = method(A, topk_per_column=topk, summation="device", **kw)
    want = pyoracle.run(family, name, A, topk_per_column=topk, order=pyoracle.ORDER_DEVICE, **kw)
    assert_same_result(got, want, f"{family}.{name} {operator} top-{topk}")
    assert np.all(np.isfinite(got.history["residual_norm"]))


# masks of one entry, of a few and of many entries a column (a thread per entry, or a warp per column), against
# columns of R that the bitmap holds and columns spread over more rows than it takes
@pytest.mark.parametrize("operator,per_column", [("diffusion", 1), ("diffusion", 20), ("diffusion", 60), ("spread", 20),
                                                 ("spread", 34)])
def test_masked_products_match_the_oracle(require_gpu, operator, per_column):
    from scipy import sparse

    from oracle import adjoint_oracle
    from parallellocallyoptimalapproximatesparsematrixinverses_b200 import adjoint
    if operator == "diffusion":
        A = problems.diffusion_2d(45, 1.0, 3)
    else:
        A = problems.random_banded_spd(40_000, half_width=1, extra=1, seed=2)
    n = A.shape[0]
    rng = np.random.default_rng(per_column)
    cols = np.repeat(np.arange(n), per_column)
    rows = (cols + rng.integers(-40, 41, cols.size)) % n if operator == "diffusion" else rng.integers(0, n, cols.size)
    M = sparse.csc_matrix(sparse.coo_matrix((rng.standard_normal(cols.size), (rows, cols)), shape=(n, n)))
    M.sum_duplicates()
    M.sort_indices()
    loss, grad_m, grad_a = adjoint.residual_adjoint(A, M)
    want_loss, want_m, want_a = adjoint_oracle.residual_adjoint(A, M)
    assert loss == want_loss
    assert np.array_equal(grad_m.data.view(np.int64), want_m.view(np.int64))
    assert np.array_equal(grad_a.data.view(np.int64), want_a.view(np.int64))
