"""Products of few long columns, split into pieces over several warps, against
the oracle: one column, columns of one piece and of many, columns of very
different lengths, and about as many columns as no longer need the split."""
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
