"""Bases with NaN rows in reach of the queries, against the oracle, bit for bit.

A NaN distance leaves the reference's batch sort, and with it the pool, out of
order, and from then on only the comparator network gives the reference's
pool: no batch may be skipped, inserted or placed by rank until the pool is
sorted again."""
import numpy as np
import pytest

from test_gpu_search import _index, _mixture

pytestmark = pytest.mark.gpu


def _nan_base(n, nq, d, share, seed):
    """An integer base (exact in FP32 and on the tensor cores) whose graph is
    that of the clean rows; `share` of its rows then hold a NaN in their last
    dimension, which the kd-tree (first three) does not read."""
    from rt_entry_gb300 import datasets as ds
    base, q = _mixture(n, nq, d, True, seed=seed)
    graph = ds.knn_graph(base, 64, device="cpu")
    rng = np.random.Generator(np.random.Philox(seed + 1))
    bad = base.copy()
    bad[rng.choice(n, int(share * n), replace=False), d - 1] = np.nan
    return bad, q, graph


# beam, width, degree, entry mode
CASES = [
    (16, 1, 64, 1), (16, 1, 16, 0), (32, 1, 64, 1), (32, 2, 32, 0), (64, 1, 64, 1), (64, 4, 16, 1),
    (128, 1, 64, 1), (128, 4, 32, 0), (256, 1, 64, 1), (256, 4, 64, 0),
]


@pytest.mark.parametrize("team", [1, 8])
@pytest.mark.parametrize("share", [0.004, 0.05])
@pytest.mark.parametrize("L,W,R,mode", CASES)
def test_nan_rows_match_oracle(lib, orc, cuda, L, W, R, mode, share, team):
    base, q, graph = _nan_base(2500, 400, 96, share, seed=23)
    graph = np.ascontiguousarray(graph[:, :R])
    idx = _index(base, graph, 24, 0.2)
    _, _, pids = idx.kdtree()
    kw = dict(search_width=W, entry_mode=mode)
    ids, dd = idx.search_projected(q, beam=L, k=L, team_warps=team, **kw)
    oids, od = orc.search(base, q, graph, L=L, k=L, leaf_pids=pids, hits=idx.locate(q), **kw)
    assert np.array_equal(ids, oids), f"{(ids != oids).any(1).sum()} queries differ"
    assert np.array_equal(dd, od)
    if mode == 1:  # leaves hold each row once: no id may come back twice
        for row in ids:
            row = row[row < len(base)]
            assert len(set(row.tolist())) == len(row)


@pytest.mark.parametrize("L", [16, 32, 64, 128])
@pytest.mark.parametrize("prec", ["bf16", "fp8"])
def test_nan_rows_in_reduced_precision(lib, orc, cuda, prec, L):
    import rt_entry_gb300 as r
    precision = {"bf16": r.PREC_BF16, "fp8": r.PREC_FP8}[prec]
    base, q, graph = _nan_base(2500, 400, 96, 0.02, seed=29)
    idx = _index(base, graph, 24, 0.2)
    _, _, pids = idx.kdtree()
    low = idx.search_base_lowp(precision)
    assert np.array_equal(np.isnan(low).any(1), np.isnan(base).any(1))
    ids, dd = idx.search_projected(q, beam=L, k=L, precision=precision)
    oids, od = orc.search(low, q, graph, L=L, k=L, leaf_pids=pids, hits=idx.locate(q))
    assert np.array_equal(ids, oids), f"{(ids != oids).any(1).sum()} queries differ"
    assert np.array_equal(dd, od)
