"""Clips whose cuts take whole faces with them, and searches that go through the weights' pyramid, against the oracle
(the same bars as test_gpu_cells.py)."""
import numpy as np
import pytest

import sdot
from test_gpu_cells import _compare, _pd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("layers", [1, 2, 5])
def test_nested_shells(d, layers):
    """a seed inside `layers` shells of 9 to 14 seeds, the outer ones met in any order: a nearer shell's cuts remove the faces
    that the farther one's made, and the vertices left over are moved"""
    rng = np.random.default_rng(10 * d + layers)
    pos = [np.full((1, d), 0.5)]
    for k in range(layers):
        u = rng.normal(size=(14 - k, d))
        pos.append(0.5 + (0.06 + 0.05 * k) * u / np.linalg.norm(u, axis=1)[:, None])
    pos.append(rng.uniform(size=(40, d)))
    pos = np.concatenate(pos)
    _compare(pos[rng.permutation(len(pos))], None)


@pytest.mark.parametrize("n", [33, 1000, 9001])
@pytest.mark.parametrize("d", [2, 3])
def test_steep_weights(d, n):
    """weights half way to those of a map onto a fraction of the box, with noise: the global bound reaches far past the rings
    and shells, so the pyramid is walked"""
    rng = np.random.default_rng(n + d)
    pos = rng.uniform(size=(n, d))
    w = 0.5 * ((pos - 0.3) ** 2).sum(axis=1) + 0.05 * n ** (-2 / d) * rng.uniform(size=n)
    _compare(pos, w)


def test_facets_come_in_the_order_met():
    """a row's neighbours come in the order the search meets them, whatever the order they cut in: by rings (2D: around the
    polygon) and, in 3D, shells of grid cells"""
    n = 4000
    pos = np.random.default_rng(5).uniform(size=(n, 3))
    nb, ids, _ = _pd(pos).hessian_rows()
    g = np.ceil(1 / (2 / n) ** (1 / 3) * (1 - 1e-12)).astype(int)
    lo, hi = np.minimum(pos.min(axis=0), 0), np.maximum(pos.max(axis=0), 1)
    cell = np.clip(((pos - lo) / ((hi - lo) / g)).astype(int), 0, g - 1)
    for i in range(0, n, 97):
        shell = np.abs(cell[ids[i, : nb[i]]] - cell[i]).max(axis=1)
        assert (np.diff(shell) >= 0).all(), (i, shell)


@pytest.mark.parametrize("others", [300, 3400])
@pytest.mark.parametrize("sides", [15, 16, 17, 31, 32, 33, 40])
def test_gaussian_cells_in_two_passes(sides, others):
    """under gaussians the cells of a diagram of 2500 seeds and more with facets are stored between two passes up to 16 vertices,
    done again past them, queued past 32; those of fewer seeds are done whole: their masses are the bits of the diagram without facets, and all is the oracle's"""
    rng = np.random.default_rng(sides)
    t = 2 * np.pi * (np.arange(sides) + 0.1 * rng.uniform(size=sides)) / sides
    ring = 0.5 + 0.2 * np.stack([np.cos(t), np.sin(t)], axis=1)
    far = rng.uniform(size=(others, 2))
    far = far[np.linalg.norm(far - 0.5, axis=1) > 0.28]
    pos = np.concatenate([far[:100], [[0.5, 0.5]], ring, far[100:]])
    c, s = rng.uniform(0.2, 0.8, (3, 2)), rng.uniform(0.1, 0.3, 3)
    g = sdot.SumOfGaussians(c, s, support_box=(np.zeros(2), np.ones(2)))
    _compare(pos, None, (("gauss", c, s, g.normalized_version().weights), g))
    args = (pos, np.zeros(len(pos)), np.zeros(2), np.ones(2), _pd(pos, dist=g)._density())
    with_facets, whole = sdot._lib.cells(*args, want_facets=True), sdot._lib.cells(*args)
    assert (with_facets["masses"] == whole["masses"]).all()
    assert with_facets["nb_count"][min(100, len(far))] == sides


@pytest.mark.parametrize("d,n,kind", [(2, n, kind) for n in (1, 700, 20011) for kind in ("uniform", "gauss", "image", "ring")] +
                         [(3, 700, "uniform"), (3, 700, "gauss")])
def test_the_rest_of_a_row_is_empty(d, n, kind):
    """past its count a row of the neighbour tables reads (-1, 0, 0), whatever the cell waited in between two passes"""
    rng = np.random.default_rng(n + d)
    pos, dist = rng.uniform(size=(n, d)), None
    if kind in ("gauss", "ring"):
        dist = sdot.SumOfGaussians(rng.uniform(0.2, 0.8, (3, d)), rng.uniform(0.1, 0.3, 3), support_box=(np.zeros(d), np.ones(d)))
    if kind == "image":
        dist = sdot.Image(rng.uniform(0.1, 1.0, size=(16, 16)), frame=[1 / 16, 1 / 16])
    if kind == "ring" and n > 1:                           # a cell of 40 edges (queued) and its neighbours of few
        t = 2 * np.pi * np.arange(40) / 40
        pos[0], pos[1:41] = 0.5, 0.5 + 0.2 * np.stack([np.cos(t), np.sin(t)], axis=1)
        pos = pos[(np.arange(n) < 41) | (np.linalg.norm(pos - 0.5, axis=1) > 0.28)]
    nb, ids, coef, meas = _pd(pos, dist=dist).facets()
    past = np.arange(ids.shape[1]) >= nb[:, None]
    assert (ids[past] == -1).all() and (coef[past] == 0).all() and (meas[past] == 0).all()
    assert (ids[~past] >= 0).all() and (coef[~past] > 0).all()
    nb, ids, coef = _pd(pos, dist=dist).hessian_rows()
    past = np.arange(ids.shape[1]) >= nb[:, None]
    assert (ids[past] == -1).all() and (coef[past] == 0).all()


@pytest.mark.parametrize("jitter", [1e-15, 4e-15, 1e-14])
@pytest.mark.parametrize("lattice", ["cubic", "face-centred"])
def test_lattices_jittered_at_the_rounding(lattice, jitter):
    """ties that rounding decides one by one.  A face moves by at most the jitter and the tie band (32 eps of lengths under 2), so a
    cell of side h changes by 12 faces times (jitter + 3e-14) / h of its volume at most; the cells cover the box"""
    m = 12
    h = 1 / m
    i = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    if lattice == "face-centred":
        i = i[i.sum(axis=1) % 2 == 0]
    rng = np.random.default_rng(len(i))
    pos = (i + 0.5) * h + rng.uniform(-jitter, jitter, size=i.shape)
    v = _pd(pos).measures
    inner = ((i > 0) & (i < m - 1)).all(axis=1)
    want = h ** 3 if lattice == "cubic" else 2 * h ** 3
    bound = 12 * (jitter + 3e-14) / h
    assert np.abs(v[inner] / want - 1).max() <= bound
    assert abs(v.sum() - 1) <= bound
