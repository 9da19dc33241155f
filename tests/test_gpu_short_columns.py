"""Products of few long columns, split into pieces over several warps, against
the oracle: one column, columns of one piece and of many, columns of very
different lengths, and about as many columns as no longer need the split; many
long columns; and many short columns beside a few long rows and columns."""
import numpy as np
import pytest
from scipy import sparse

from oracle import pyoracle
from parallellocallyoptimalapproximatesparsematrixinverses_b200 import global_spai, problems
from tests.helpers import assert_same_result

pytestmark = pytest.mark.gpu


def _dense(n):
    a = np.random.default_rng(n).uniform(-0.5, 0.5, (n, n))
    return sparse.csc_matrix((a + a.T) * 0.5 + n * np.eye(n))


def _uneven(n):
    """A dense corner beside a diagonal: columns of n / 4 entries and of one."""
    a = sparse.lil_matrix((n, n))
    k = n // 4
    a[:k, :k] = _dense(k)
    a.setdiag(n)
    return sparse.csc_matrix(a)


OPERATORS = {"dense_1": lambda: _dense(1), "dense_31": lambda: _dense(31), "dense_97": lambda: _dense(97),
             "dense_333": lambda: _dense(333), "uneven_1300": lambda: _uneven(1300), "uneven_1775": lambda: _uneven(1775),
             "uneven_1776": lambda: _uneven(1776)}


@pytest.mark.parametrize("operator", sorted(OPERATORS))
def test_products_of_few_long_columns_match_the_oracle(require_gpu, operator):
    A = OPERATORS[operator]()
    kw = dict(M0=problems.diagonal_inverse(A), max_iterations=2, tolerance=0.0, max_density=1.0, enable_dropping=False)
    got = global_spai.mr(A, summation="device", **kw)
    want = pyoracle.run("global_spai", "mr", A, order=pyoracle.ORDER_DEVICE, **kw)
    assert_same_result(got, want, operator)


def _arrow(n):
    hub = n // 3
    a = sparse.lil_matrix((n, n))
    a[hub, :] = a[:, hub] = np.linspace(0.1, 0.9, n)
    a.setdiag(2.0 * n)
    a = sparse.csc_matrix(a)
    return sparse.csc_matrix((a + a.T) * 0.5)


# a column of A beyond 2,048 entries sends every product down the generic way: residuals of two entries a column, and
# products with Z and P whose columns are all full
@pytest.mark.parametrize("method,n,topk", [("mr", 2500, 2), ("lomr", 2500, 3), ("cg", 2500, 2), ("mr", 8500, 4)])
def test_products_around_a_long_row_match_the_oracle(require_gpu, method, n, topk):
    A = _arrow(n)
    kw = dict(M0=problems.diagonal_inverse(A), max_iterations=2 if n < 8000 else 1, tolerance=0.0, max_density=topk / n,
              topk_per_column=topk)
    got = getattr(global_spai, method)(A, summation="device", **kw)
    want = pyoracle.run("global_spai", method, A, order=pyoracle.ORDER_DEVICE, **kw)
    assert_same_result(got, want, f"{method} {n}")
