"""The Laplacian's rows, made by several lanes each, against the facets of the diagram."""
import numpy as np
import pytest

from test_gpu_cells import _pd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(2, 2), (2, 63), (2, 64), (2, 65), (2, 257), (3, 9), (3, 257), (2, 40), (2, 41)])
def test_the_rows_are_the_mutual_facets(d, n):
    """sizes around a chunk's rows; (2, 40) and (2, 41): a seed inside a ring, its row of more than 32 facets in the overflow
    store.  Entries in facet order, the two of a pair the same bits (the lower row's), the diagonal their sum in that order"""
    rng = np.random.default_rng(n)
    pos = rng.uniform(size=(n, d))
    if n in (40, 41):
        t = 2 * np.pi * np.arange(1, n) / (n - 1) + 0.01 * rng.uniform(size=n - 1)
        pos[0], pos[1:] = 0.5, 0.5 + 0.3 * np.stack([np.cos(t), np.sin(t)], axis=1)
        pos[[0, n // 2]] = pos[[n // 2, 0]]
    nb, ids, val = _pd(pos).hessian_rows()
    rows = [dict(zip(ids[i, : nb[i]], val[i, : nb[i]])) for i in range(n)]
    row_ptr, cols, vals, dia = _pd(pos).laplacian()
    assert max(nb) > 32 or n not in (40, 41)
    for i in range(n):
        want = [(j, rows[min(i, j)][max(i, j)]) for j in rows[i] if i in rows[j]]
        got = list(zip(cols[row_ptr[i] : row_ptr[i + 1]], vals[row_ptr[i] : row_ptr[i + 1]]))
        assert got == want
        assert dia[i] == (sum((c for _, c in want), 0.0) or 1.0)
