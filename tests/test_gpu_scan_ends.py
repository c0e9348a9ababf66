"""Queued scans of dense cells end where their part of the cell ends, also
where eps squared leaves float's range: layouts in which a point counted twice,
or a point of the next cell taken for one of this cell, changes a label."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCALES = [1.0, 1e-22, 1e19, 1e22, 1e30]
DENSE = 1500  # points of a dense cell, above the length at which a scan is queued


def _side(d):
    """Cell side for eps = 1."""
    return 1.0 / np.sqrt(d)


@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("scale", SCALES)
def test_count_of_a_queued_scan(engine, oracle, d, scale):
    """A stray reaches about half of a dense cell, too few to be core, so that a
    point near the stray alone is noise."""
    rng = np.random.default_rng(d)
    s = _side(d)
    dense = rng.uniform(0.02, 0.98, size=(DENSE, d)) * s
    stray = np.full(d, 0.5 * s)
    stray[0] = 0.5 * s + 1.0
    reach = np.linalg.norm(dense - stray, axis=1)
    stray[0] += np.median(reach) - 1.0  # the median point is now about eps away
    reach = int((np.linalg.norm(dense - stray, axis=1) < 1.0).sum())
    min_pts = 1200
    assert 400 < reach + 1 < min_pts
    beyond = stray.copy()
    beyond[0] += 0.9
    X = np.concatenate([dense, [stray, beyond]])
    order = np.random.default_rng(7).permutation(len(X))
    lab = engine.dbscan(X[order] * scale, scale, min_pts)
    assert np.array_equal(lab, oracle.dbscan(X[order] * scale, scale, min_pts))
    back = np.empty_like(lab)
    back[order] = lab
    assert (back[:DENSE] == 0).all() and back[DENSE] == 0 and back[DENSE + 1] == -1


@pytest.mark.parametrize("scale", SCALES)
def test_labels_of_a_queued_scan(engine, oracle, scale):
    """A border point near two dense cells, one of which has its box but no
    point within eps: it takes the other's label, whichever of the cells' points
    come first in memory."""
    rng = np.random.default_rng(0)
    s = _side(2)
    X, at, kind = [], [], []
    for k in range(16):  # 16 copies far apart, in all directions
        turn = np.array([[1, 0], [0, 1]])[:, :: (-1 if k & 4 else 1)] * [1 if k & 1 else -1, 1 if k & 2 else -1]
        corners = np.where(rng.random((DENSE, 1)) < 0.5, [[0.08, 0.92]], [[0.92, 0.08]])
        empty = corners + rng.uniform(-0.05, 0.05, size=(DENSE, 2))
        full = rng.uniform(2.15, 2.95, size=(DENSE, 2))
        border = np.array([[1.6, 1.6]])
        near = np.linalg.norm(full - border, axis=1) * s < 1.0
        assert 100 < near.sum() < 1200
        far = full[~near]
        full = np.concatenate([far[::2], full[near], far[1::2]])  # first and last (representatives) out of reach
        assert np.linalg.norm(empty - border, axis=1).min() * s > 1.0
        origin = np.array([20.0 * k, 11.0 * (k % 5)])
        # mirrored about the middle of cell 1, so that cells stay whole cells
        X.append(((np.concatenate([empty, full, border]) - 1.5) @ turn + 1.5 + origin) * s)
        kind += [0] * DENSE + [1] * DENSE + [2]
    X, kind = np.concatenate(X), np.array(kind)
    lab = engine.dbscan(X * scale, scale, 1400)
    assert np.array_equal(lab, oracle.dbscan(X * scale, scale, 1400))
    per = 2 * DENSE + 1
    for k in range(16):
        mine = lab[per * k: per * (k + 1)]
        assert mine[0] >= 0 and mine[-1] == mine[DENSE] != mine[0], k
