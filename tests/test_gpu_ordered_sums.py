"""Sums in the reference's order of several long column batches (each over
16,384 entries: eight blocks a batch), several tiles long and ending inside a
piece, against the oracle."""
import pytest

from oracle import pyoracle
from parallellocallyoptimalapproximatesparsematrixinverses_b200 import global_spai, problems
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
