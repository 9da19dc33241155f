"""Which kernels a fused Global MR run takes (read from the library's own
accounting), and the same bits as the unfused kernels on each way."""
import ctypes

import numpy as np
import pytest
from scipy import sparse

from parallellocallyoptimalapproximatesparsematrixinverses_b200 import Session, _lib, global_spai, problems
from tests.helpers import assert_same_result

pytestmark = pytest.mark.gpu


def _launches(lib, name):
    ms, count, nbytes = ctypes.c_double(0), ctypes.c_int64(0), ctypes.c_double(0)
    lib.spai_profile_read(name.encode(), ctypes.byref(ms), ctypes.byref(count), ctypes.byref(nbytes))
    return count.value, nbytes.value


def profiled(call, *names):
    """call()'s result and the launches and algorithmic bytes of the named kernel classes."""
    lib = _lib.load()
    lib.spai_profile_reset()
    lib.spai_profile_enable(1)
    try:
        result = call()
    finally:
        lib.spai_profile_enable(0)
    counts = {name: _launches(lib, name) for name in names}
    lib.spai_profile_reset()
    return result, counts


def unfused(call):
    lib = _lib.load()
    lib.spai_set_fused_mr(0)
    try:
        return call()
    finally:
        lib.spai_set_fused_mr(1)


def band(n, distances, seed=0):
    """Symmetric, diagonally dominant, entries at the given distances from the diagonal."""
    rng = np.random.default_rng(seed)
    rows = np.concatenate([np.arange(n - d) for d in distances])
    cols = np.concatenate([np.arange(n - d) + d for d in distances])
    off = sparse.coo_matrix((-rng.uniform(0.1, 1.0, rows.size), (rows, cols)), shape=(n, n)).tocsr()
    off = off + off.T
    a = sparse.csc_matrix(off + sparse.diags(1.05 * np.asarray(abs(off).sum(axis=1)).ravel() + 0.1))
    a.sort_indices()
    return a


# operators wider than any window of a column group, rows of A in 4, 8, 12 and 16 slots
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("distances,topk", [([9000], 6), ([1, 9000], 8), ([1, 2, 3, 9000], 5), ([1, 2, 3, 4, 5, 9000], 5)])
def test_wide_operators_run_on_the_column_kernels(require_gpu, distances, topk, precision):
    a = band(18_011, distances)
    kw = dict(M0=problems.diagonal_inverse(a), max_iterations=7, tolerance=0.0, max_density=topk / a.shape[0],
              topk_per_column=topk, precision=precision)
    got, counts = profiled(lambda: global_spai.mr(a, **kw), "fused_drop", "fused_drop_columns", "fused_residual",
                           "fused_residual_columns")
    assert counts["fused_drop"][0] == counts["fused_residual"][0] == 0
    assert counts["fused_drop_columns"][0] == counts["fused_residual_columns"][0] == 7
    want = unfused(lambda: global_spai.mr(a, **kw))
    assert_same_result(got, want, f"{distances} {precision}, launched one by one")
    assert_same_result(global_spai.mr(a, **kw), want, f"{distances} {precision}, as a graph")


def shuffled(a, span, seed=1):
    """Rows and columns permuted within blocks of `span`: adjacent columns share no rows, inside the window."""
    n = a.shape[0]
    rng = np.random.default_rng(seed)
    p = np.concatenate([lo + rng.permutation(min(span, n - lo)) for lo in range(0, n, span)])
    a = sparse.csc_matrix(a[p][:, p])
    a.sort_indices()
    return a


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_scattered_columns_leave_the_groups(require_gpu, precision):
    a = shuffled(problems.diffusion_3d(22, 1.0, 5), 2000)
    topk = 20
    kw = dict(M0=problems.diagonal_inverse(a), max_iterations=8, tolerance=0.0, max_density=topk / a.shape[0],
              topk_per_column=topk, precision=precision)
    want = unfused(lambda: global_spai.mr(a, **kw))
    got, counts = profiled(lambda: global_spai.mr(a, **kw), "fused_drop", "fused_drop_columns")
    # the first steps' columns are short enough for groups, the later ones are not
    assert counts["fused_drop"][0] > 0 and counts["fused_drop_columns"][0] > 0
    assert counts["fused_drop"][0] + counts["fused_drop_columns"][0] == 8
    assert_same_result(got, want, f"{precision}, launched one by one")
    assert_same_result(global_spai.mr(a, **kw), want, f"{precision}, as graphs")
    # a second run on the same problem starts column by column
    session = Session("global_spai", "mr", a, **kw)
    session.run()
    first = session.result()
    _, counts = profiled(session.run, "fused_drop", "fused_drop_columns")
    assert counts["fused_drop"][0] == 0 and counts["fused_drop_columns"][0] == 8
    assert_same_result(first, want, f"{precision}, first run")
    assert_same_result(session.result(), want, f"{precision}, second run")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_scattered_systems_of_a_batch_leave_the_groups(require_gpu, precision):
    batch = [shuffled(problems.diffusion_3d(22, 1.0, 5), 2000), problems.diffusion_2d(30, 1.0, 2)]
    kw = dict(max_iterations=7, tolerance=0.0, max_density=1.0, topk_per_column=20, precision=precision)
    want = unfused(lambda: global_spai.mr_batched(batch, **kw))
    got, counts = profiled(lambda: global_spai.mr_batched(batch, **kw), "fused_drop", "fused_drop_columns")
    assert counts["fused_drop"][0] > 0 and counts["fused_drop_columns"][0] > 0
    for b, (g, w) in enumerate(zip(got, want)):
        assert_same_result(g, w, f"{precision} system {b}")


def test_grids_stay_in_groups(require_gpu):
    a = problems.diffusion_3d(22, 1.0, 5)
    kw = dict(M0=problems.diagonal_inverse(a), max_iterations=8, tolerance=0.0, max_density=16 / a.shape[0],
              topk_per_column=16)
    _, counts = profiled(lambda: global_spai.mr(a, **kw), "fused_drop", "fused_drop_columns")
    assert counts["fused_drop"][0] == 8 and counts["fused_drop_columns"][0] == 0


def tree(degree, depth):
    """A tree's graph Laplacian, slightly shifted: the row of M at its root grows with every step."""
    parent, frontier = [-1], [0]
    for _ in range(depth):
        grown = []
        for p in frontier:
            for _ in range(degree if p == 0 else degree - 1):
                parent.append(p)
                grown.append(len(parent) - 1)
        frontier = grown
    n = len(parent)
    off = sparse.coo_matrix((-np.ones(n - 1), (np.arange(1, n), parent[1:])), shape=(n, n)).tocsr()
    off = off + off.T
    a = sparse.csc_matrix(off + sparse.diags(1.02 * np.asarray(abs(off).sum(axis=1)).ravel()))
    a.sort_indices()
    return a


# the root's row of M has 5, 15 and 44 entries after the first steps, its slots are 32: the third step is void
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_batch_goes_on_from_the_step_that_outgrew_its_slots(require_gpu, precision):
    batch = [problems.diffusion_2d(19, 0.5, 3), tree(4, 5), problems.tridiagonal(40)]
    kw = dict(max_iterations=7, tolerance=0.0, max_density=1.0, topk_per_column=8, precision=precision)
    names = ("fused_drop", "union")
    want, unfused_counts = unfused(lambda: profiled(lambda: global_spai.mr_batched(batch, **kw), *names))
    got, counts = profiled(lambda: global_spai.mr_batched(batch, **kw), *names)
    assert counts["fused_drop"][0] == 3
    per_step = unfused_counts["union"][0] // 7
    assert per_step >= 1 and unfused_counts["union"][0] - counts["union"][0] == 2 * per_step
    for b, (g, w) in enumerate(zip(got, want)):
        assert_same_result(g, w, f"{precision} system {b}")


def test_batched_steps_account_for_their_bytes(require_gpu):
    """A batch of one system moves what the system alone moves."""
    a = problems.diffusion_2d(40, 0.5, 3)
    kw = dict(max_iterations=6, tolerance=0.0, max_density=1.0, topk_per_column=8)
    names = ("fused_drop", "fused_residual")
    _, alone = profiled(lambda: global_spai.mr(a, **kw), *names)
    _, batch = profiled(lambda: global_spai.mr_batched([a], **kw), *names)
    for name in names:
        assert alone[name][0] == batch[name][0] == 6
        assert alone[name][1] == batch[name][1] > 0


# the largest cap and the longest rows the fused kernels take, in groups of four
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", ["top_32", "rows_of_13", "rows_of_9"])
def test_the_largest_groups_run_fused(require_gpu, case, precision):
    a, topk = {"top_32": lambda: (problems.diffusion_2d(101, 1.0, 5), 32),
               "rows_of_13": lambda: (band(9_999, [1, 2, 3, 40, 41, 90]), 5),
               "rows_of_9": lambda: (band(9_999, [1, 2, 50, 51]), 12)}[case]()
    kw = dict(M0=problems.diagonal_inverse(a), max_iterations=9, tolerance=0.0, max_density=topk / a.shape[0],
              topk_per_column=topk, precision=precision)
    want = unfused(lambda: global_spai.mr(a, **kw))
    got, counts = profiled(lambda: global_spai.mr(a, **kw), "fused_drop", "fused_drop_columns", "drop_update")
    assert counts["fused_drop"][0] + counts["fused_drop_columns"][0] == 9
    assert counts["fused_drop"][0] >= 1 and counts["drop_update"][0] == 1
    assert_same_result(got, want, f"{case} {precision}")


# an entry of A beyond FP32's range: the column groups would multiply it by the 0 of an absent entry
def test_a_system_that_is_not_finite_in_fp32_storage(require_gpu):
    bad = problems.diffusion_2d(20, 1.0, 4).tolil()
    bad[7, 8] = bad[8, 7] = 1e39
    batch = [problems.diffusion_2d(31, 1.0, 2), sparse.csc_matrix(bad), problems.diffusion_3d(9, 1.0, 1)]
    kw = dict(max_iterations=6, tolerance=0.0, max_density=1.0, topk_per_column=6, precision="mixed")
    want = unfused(lambda: global_spai.mr_batched(batch, **kw))
    got, counts = profiled(lambda: global_spai.mr_batched(batch, **kw), "fused_drop", "fused_drop_columns")
    assert counts["fused_drop"][0] == 0 and counts["fused_drop_columns"][0] >= 1
    for b, (g, w) in enumerate(zip(got, want)):
        assert_same_result(g, w, f"system {b}")
    assert not np.isfinite(got[1].history["residual_norm"][0]) and np.all(np.isfinite(got[0].history["residual_norm"]))
