"""The clustering's block tables and queued long scans against the oracle:
more distinct cells per block than its table holds, and thousands of
undecided points around cells of more than 1,024 points, some queueing a scan
of several such cells each (more than the queue holds), with the minimum
number of points below and above what one cell gives; pairs of cells with
thousands of points that just do or do not reach each other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d, n", [(1, 1500), (2, 30000), (3, 30000)])
def test_many_cells_per_block(engine, oracle, d, n):
    X = np.random.default_rng(d).uniform(0, 1, size=(n, d))
    eps = 0.3 / n ** (1.0 / d)  # nearly every point in a cell of its own
    assert np.array_equal(engine.dbscan(X, eps, 2), oracle.dbscan(X, eps, 2))


@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("min_pts", [3, 1200, 2500])
@pytest.mark.parametrize("scale", [1.0, 1e-22, 1e22])  # the last two leave float's range when squared
def test_long_scans(engine, oracle, d, min_pts, scale):
    rng = np.random.default_rng(10 * d + min_pts)
    eps = 0.05
    side = eps / d ** 0.5
    centres = (np.stack(np.meshgrid(*[np.arange(2)] * d), -1).reshape(-1, d) + 0.5) * side
    blobs = np.concatenate([c + rng.uniform(-0.3, 0.3, size=(1500, d)) * side for c in centres])
    strays = rng.uniform(-1.2, 3.2, size=(7000, d)) * side
    strays = strays[(np.abs(strays / side - 1.0) > 1.0).any(axis=1)]
    X = np.concatenate([blobs, strays])
    X = X[rng.permutation(len(X))] * scale
    lab = engine.dbscan(X, eps * scale, min_pts)
    ref = oracle.dbscan(X, eps * scale, min_pts)
    assert np.array_equal(lab, ref)


@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("few", [3, 300, 2000])
@pytest.mark.parametrize("gap", [0.99999, 1.0, 1.00001])
def test_long_pairs(engine, oracle, d, few, gap):
    """Two groups whose nearest points are eps * gap apart, in cells whose
    boxes do not settle it: joined exactly when a pair is within eps."""
    rng = np.random.default_rng(d)
    eps = 0.05
    a = rng.uniform(-0.2, 0.0, size=(4000, d)) * eps
    b = rng.uniform(0.0, 0.2, size=(few, d)) * eps
    a[:, 1:] = rng.uniform(-0.3, 0.3, size=(4000, d - 1)) * eps
    b[:, 1:] = rng.uniform(-0.3, 0.3, size=(few, d - 1)) * eps
    a[17], b[1] = 0.0, 0.0
    b[:, 0] += eps * gap
    X = np.concatenate([a, b])
    X = X[rng.permutation(len(X))] + 0.5
    for min_pts in (2, few, 3000):
        lab = engine.dbscan(X, eps, min_pts)
        ref = oracle.dbscan(X, eps, min_pts)
        assert np.array_equal(lab, ref), min_pts
