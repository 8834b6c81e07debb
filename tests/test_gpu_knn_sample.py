"""The kNN builder's threshold sample: rows of every group of a base whose
groups come in turns, whatever the period."""
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _left(capfd):
    """Rows that the thresholded pass left to the stored products."""
    m = re.search(r"(\d+) rows in memory", capfd.readouterr().err)
    assert m
    return int(m.group(1))


@pytest.mark.parametrize("n,period", [(24000, 24), (24000, 8), (24000, 2), (6143, 23)])
def test_groups_in_turns_keep_to_the_pass(lib, cuda, capfd, monkeypatch, n, period):
    import rt_entry_gb300 as r
    from rt_entry_gb300 import datasets as ds
    rng = np.random.Generator(np.random.Philox(period))
    base = (100 * rng.random((period, 32))[np.arange(n) % period]
            + 5 * rng.standard_normal((n, 32))).astype(np.float32)
    monkeypatch.setenv("RTE_KNN_VERBOSE", "1")
    g = r.knn_graph(base, 32)
    assert _left(capfd) <= n // 100
    rows = rng.choice(n, 500, replace=False)
    wide = base.astype(np.float64)
    d2 = np.stack([((wide - wide[i]) ** 2).sum(1) for i in rows])
    d2[np.arange(500), rows] = np.inf
    want = np.stack([np.lexsort((np.arange(n), v))[:32] for v in d2])
    assert np.array_equal(g[rows], want)
