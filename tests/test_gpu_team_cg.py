"""The FP64 CG of one launch (a team of blocks per system) at the sizes where its cut of the rows changes: one share, the
first row of the next, the largest cluster, the first cooperative team, one share more than it has rows for.

The solution is held by its true residual.  The CG stops at |r| <= tol |b| on the residual it updates; that one and b - L x
drift apart by at most a few eps |L| |x| an iteration (each iteration's x and r are rounded once), so
|b - L x| <= tol |b| + 4 eps its |L|_inf |x|."""
import numpy as np
import pytest
import scipy.sparse as sp

from sdot import _lib

pytestmark = pytest.mark.gpu


def ring(n, seed):
    """the Laplacian of n seeds on a ring, each tied to its nearest two and one at distance 7, couplings in [0.5, 2]"""
    rng = np.random.default_rng(seed)
    i = np.concatenate([np.arange(n)] * 3)
    j = np.concatenate([(np.arange(n) + k) % n for k in (1, 2, 7)])
    c = rng.uniform(0.5, 2.0, size=len(i))
    keep = i != j
    A = sp.coo_matrix((c[keep], (i[keep], j[keep])), shape=(n, n)).tocsr()
    A = (A + A.T).tocsr()
    A.sum_duplicates()
    return A, np.asarray(A.sum(axis=1)).reshape(-1)


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("n", [9, 32, 33, 128, 129, 2048, 2049, 18944, 18945])
def test_residual(n, method):
    A, dia = ring(n, n)
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
    assert _lib.linear_solve(A.indptr, A.indices, A.data, dia, b, tol=tol, maxit=3, method=method)[1][0] in (-1, 1, 2, 3)
