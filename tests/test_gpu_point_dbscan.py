"""The per-point interval clustering against the oracle at the edges of its
bit words: rows around multiples of 32 entries, the longest row kept as bits
(1,024) and the first one kept in scratch, with intervals in few groups, in
many, all alike, and with infinite and undefined entries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 31, 32, 33, 34, 63, 64, 65, 66, 97, 500, 1023, 1024, 1025, 1026, 1100]


@pytest.mark.parametrize("kind", ["alike", "groups", "spread", "chain", "odd"])
@pytest.mark.parametrize("eps", [0.02, 0.0, float("inf")])
def test_rows_at_word_edges(engine, oracle, kind, eps):
    rng = np.random.default_rng(5)
    rows = [p for p in SIZES for _ in range(6)]
    iv = np.zeros((len(rows), max(SIZES)))
    for r, p in enumerate(rows):
        v = {
            "alike": lambda: np.full(p, 1.25),
            "groups": lambda: np.round(rng.uniform(0, 1, p) * 8) / 8 + rng.uniform(-0.012, 0.012, p),
            "spread": lambda: rng.uniform(0, 0.15 * p, p),
            "chain": lambda: rng.permutation(np.arange(p) * rng.choice([0.0199, 0.02, 0.0201])),
            "odd": lambda: rng.choice([0.0, -0.0, 0.01, np.inf, -np.inf, np.nan, 1e300, 5e-324], p),
        }[kind]()
        iv[r, :p] = v
    counts = np.array(rows, dtype=np.int32)
    assert np.array_equal(engine.point_dbscan(iv, counts, eps), oracle.point_dbscan(iv, counts, eps))
