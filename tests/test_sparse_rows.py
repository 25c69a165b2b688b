"""The batched sparse solve's two routes on a B200 (a block's shared memory, or the level launches for factors past a block),
at the smallest sizes, around a group of 32 systems and past a block: solutions come back in the order of the unknowns,
systems of alternating patterns, values that collapse a static pivot, right-hand sides that are not finite. Residuals within
1e-12 of |A| |x| + |b|, row by row (diagonally dominant systems: a few hundred roundings of 2.2e-16)."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _matrix(n, seed):
    rng = np.random.default_rng(seed)
    a = sp.diags([rng.uniform(-1, 1, n) for _ in range(3)], [-1, 0, 1], shape=(n, n), format="lil")
    for i in rng.integers(0, n, size=n // 3):
        a[i, min(n - 1, i + rng.integers(2, 12))] = rng.uniform(-1, 1)
    a = sp.csr_matrix(a)
    a = a + sp.diags(np.asarray(abs(a).sum(axis=1)).ravel() + 1.0, format="csr")
    a.sort_indices()
    return a


def _near(a, x, b):
    return (np.abs(a @ x - b) <= 1e-12 * (abs(a) @ np.abs(x) + np.abs(b))).all()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1500, 12000])
@pytest.mark.parametrize("count", [1, 33])
def test_rows(n, count):
    from gridsim_b200.engine import CudaSparseLinearSolver
    base = _matrix(n, n)
    rng = np.random.default_rng(n + count)
    mats = [sp.csr_matrix((base.data * rng.uniform(0.9, 1.0, base.nnz), base.indices, base.indptr), shape=(n, n)) for _ in range(count)]
    for m in mats:
        m.setdiag(base.diagonal())
    rhs = [rng.standard_normal(n) for _ in mats]
    for m, x, b in zip(mats, CudaSparseLinearSolver().solve_batch(mats, rhs), rhs):
        assert _near(m, x, b)


@pytest.mark.parametrize("n", [31, 1500])
def test_failures_and_other_patterns_between(n):
    from gridsim_b200.engine import CudaSparseLinearSolver
    a, other = _matrix(n, 1), _matrix(n, 2)
    singular = a.copy()
    singular.data[singular.indptr[3]:singular.indptr[4]] = 0.0
    swapped = sp.csr_matrix(([1.0, 1.0, 2.0], [1, 0, 1], [0, 1, 3]), shape=(2, 2))
    b = np.random.default_rng(3).standard_normal(n)
    bad = b.copy()
    bad[n // 2] = np.inf
    mats = [a, a, other, singular, a, swapped, a]
    rhs = [b, bad, b, b, 2 * b, np.array([1.0, 4.0]), b]
    errors = [None] * len(mats)
    xs = CudaSparseLinearSolver().solve_batch(mats, rhs, errors)
    assert isinstance(errors[1], ValueError) and xs[1] is None
    assert xs[3] is None
    for k in (0, 2, 4, 5, 6):
        assert errors[k] is None and _near(mats[k], xs[k], rhs[k]), k
    assert np.array_equal(xs[0], xs[6])
