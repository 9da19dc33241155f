"""Sums in the reference's order evaluated in parallel pieces: the arithmetic
(csrc/ordered_sum.cuh) against a plain loop on the CPU, and the kernels through
the drop-in methods against the oracle in the reference's order."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import pyoracle
from parallellocallyoptimalapproximatesparsematrixinverses_b200 import global_spai, problems
from tests.helpers import assert_same_result

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "parallellocallyoptimalapproximatesparsematrixinverses_b200" / "csrc"


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = tmp_path_factory.mktemp("ordered_sum") / "ordered_sum_test"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{CSRC}",
                    str(ROOT / "tests" / "cpp" / "ordered_sum_test.cpp"), "-o", str(out)], check=True)
    return out


@pytest.mark.parametrize("kind", range(8))
def test_pieces_give_the_loops_bits(program, kind):
    done = subprocess.run([str(program), str(kind)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
    if kind in (0, 1, 3):
        assert int(done.stdout) > 0  # summaries were used, not only the term-by-term path


# batches of one column up to the whole matrix: blocks of 32 and 256 threads and
# clusters of eight blocks, tiles that end inside a piece, sums with ties (the Laplacian's dyadic values)
@pytest.mark.gpu
@pytest.mark.parametrize("threads", [1, 2, 37, 1521])
@pytest.mark.parametrize("method", ["cg", "mr", "lomr"])
@pytest.mark.parametrize("operator", ["diffusion", "laplacian"])
def test_drop_in_sums_match_the_oracle(require_gpu, operator, method, threads):
    A = problems.diffusion_2d(39, 1.0, 5) if operator == "diffusion" else problems.laplacian_2d(39)
    kw = dict(M0=problems.diagonal_inverse(A), max_iterations=5, tolerance=1e-12, max_density=14.0 / A.shape[0],
              num_threads=threads)
    got = getattr(global_spai, method)(A, **kw)
    want = pyoracle.run("global_spai", method, A, order=pyoracle.ORDER_REFERENCE, **kw)
    assert_same_result(got, want, f"{method} {operator} {threads} threads")
    assert np.all(np.isfinite(got.history["residual_norm"]))
