"""The FP64 CG of one launch (a team of blocks per system) at the sizes where its cut of the rows changes: one share, the
first row of the next, the largest cluster, the first cooperative team, one share more than it has rows for.

The solution is held by its true residual.  The CG stops at |r| <= tol |b| on the residual it updates; that one and b - L x
drift apart by at most a few eps |L| |x| an iteration (each iteration's x and r are rounded once), so
|b - L x| <= tol |b| + 4 eps its |L|_inf |x|."""
import numpy as np
import pytest
import scipy.sparse as sp

from sdot import Box, Iterative, OtProblem, SumOfDiracs, Tuning, _lib
from sdot.SdotPlanNd import SdotPlanNd, solver_options

pytestmark = pytest.mark.gpu


def ring(n, seed, ties=(1, 2, 7)):
    """the Laplacian of n seeds on a ring, each tied to those at these distances, couplings in [0.5, 2]"""
    rng = np.random.default_rng(seed)
    i = np.concatenate([np.arange(n)] * len(ties))
    j = np.concatenate([(np.arange(n) + k) % n for k in ties])
    c = rng.uniform(0.5, 2.0, size=len(i))
    keep = i != j
    A = sp.coo_matrix((c[keep], (i[keep], j[keep])), shape=(n, n)).tocsr()
    A = (A + A.T).tocsr()
    A.sum_duplicates()
    return A, np.asarray(A.sum(axis=1)).reshape(-1)


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("n", [9, 32, 33, 128, 129, 2048, 2049, 18944, 18945])
def test_residual(n, method):
    _residual(n, method, (1, 2, 7))


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("n", [33, 128, 129, 2049, 18944, 18945, 40003])
def test_residual_of_rows_of_sixteen(n, method):
    """as many entries as a 3D Laplacian's rows: the multigrid's aggregates are of 8, a row has 8 lanes"""
    _residual(n, method, (1, 2, 3, 4, 5, 7, 11, 13))


def _residual(n, method, ties):
    A, dia = ring(n, n, ties)
    b = np.random.default_rng(n + 1).normal(size=n)
    b -= b.mean()
    tol = 1e-9
    x, its = _lib.linear_solve(A.indptr, A.indices, A.data, dia, b, tol=tol, maxit=100000, method=method)
    assert its[0] > 0
    x = x[0]
    assert x[0] == 0
    r = b - (dia * x - A @ x)
    bound = tol * np.linalg.norm(b) + 4 * np.finfo(float).eps * its[0] * 2 * dia.max() * np.linalg.norm(x)
    assert np.linalg.norm(r) <= bound, (np.linalg.norm(r), bound)
    y, its2 = _lib.linear_solve(A.indptr, A.indices, A.data, dia, b, tol=tol, maxit=100000, method=method)
    assert its2[0] == its[0] and (y[0] == x).all()              # fixed sums: the same bits
    short = _lib.linear_solve(A.indptr, A.indices, A.data, dia, b, tol=tol, maxit=3, method=method)[1][0]
    assert short == (its[0] if its[0] <= 3 else -1)             # three iterations, and no success without convergence


@pytest.mark.parametrize("others", [4, 39])
@pytest.mark.parametrize("d,n", [(2, 20011), (3, 20000), (2, 2500)])
def test_a_system_has_the_same_bits_in_any_team(d, n, others):
    """alone a block plays one share, meeting the others at a counter in memory; in a batch its team shrinks to a few blocks of many
    shares, in a cluster or not, in one of several launches: the same solve to the bit"""
    rng = np.random.default_rng(n)
    settings = Iterative(tol=0.0, tuning=Tuning(mass_rtol=1e-8))
    one = OtProblem(SumOfDiracs(rng.uniform(size=(n, d))), Box(nb_dims=d))
    sizes = rng.integers(500, 20012, size=others)
    rest = [OtProblem(SumOfDiracs(rng.uniform(size=(m, 2 + k % 2))), Box(nb_dims=2 + k % 2)) for k, m in enumerate(sizes)]
    alone = SdotPlanNd._solve_many([one], settings)[0]
    batch = SdotPlanNd._solve_many(rest[:2] + [one] + rest[2:], settings)[2]
    assert alone.stats["lin_nb_iter"] == batch.stats["lin_nb_iter"]
    assert (alone.weights == batch.weights).all() and (alone.cell_masses == batch.cell_masses).all()


def test_a_barrier_that_waits_in_vain_is_an_error():
    """with a single poll the first blocks of a team give up before the last has come: the call says so -- it is not a system that the
    CG could not solve --, and the context solves again afterwards"""
    n = 20011
    rng = np.random.default_rng(1)
    pos = rng.uniform(size=(n, 2))
    problem = (pos, None, None, np.zeros(2), np.ones(2), ("uniform", 1.0))
    options = solver_options(Iterative(tol=0.0, tuning=Tuning(mass_rtol=1e-8)), n, 2)
    L = _lib.load()
    ctx = _lib.new_context()
    try:
        before, = _lib.solve_batch([problem], [options], ctx=ctx)
        assert L.sdot_context_set_barrier_polls(ctx, 1) == _lib.SDOT_OK
        failed, = _lib.solve_batch([problem], [options], ctx=ctx)
        assert isinstance(failed, RuntimeError) and "barrier" in str(failed)
        assert L.sdot_context_set_barrier_polls(ctx, 0) == _lib.SDOT_OK
        after, = _lib.solve_batch([problem], [options], ctx=ctx)
        assert (after["weights"] == before["weights"]).all()
    finally:
        _lib.destroy_context(ctx)
    A, dia = ring(n, n)
    b = rng.normal(size=n)
    b -= b.mean()
    L.sdot_context_set_barrier_polls(_lib.context(), 1)
    try:
        for method in (0, 1):
            with pytest.raises(RuntimeError, match="barrier"):
                _lib.linear_solve(A.indptr, A.indices, A.data, dia, b, tol=1e-9, method=method)
    finally:
        L.sdot_context_set_barrier_polls(_lib.context(), 0)
    assert _lib.linear_solve(A.indptr, A.indices, A.data, dia, b, tol=1e-9)[1][0] > 0
