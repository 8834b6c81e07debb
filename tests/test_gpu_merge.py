"""The search kernel's merge and filter paths against the oracle, bit for bit.

A batch's candidates are inserted (up to 4, pools of 16 to 64), ranked (up to
32, or 64 in batches of 128 and more) and placed, or sorted by the reference's
network (more, or equal distances).  The visited filter has one path per
number of registers a neighbour list fills, and one for more than 3 hashes.
Everything is integer arithmetic or FP32 in the oracle's order, so results
are compared for equality.
"""
import numpy as np
import pytest

from test_gpu_search import _index, _mixture

pytestmark = pytest.mark.gpu

# d, degree, beam, width, data ("dup": the second half repeats the first),
# hashes, entry mode
CASES = [
    # one list fills the batch: 1, 2, 4 and 8 registers
    (128, 32, 16, 1, "real", 3, 1),
    (128, 64, 32, 1, "dup", 2, 1),
    (96, 128, 64, 1, "real", 3, 1),
    (128, 256, 256, 1, "real", 3, 1),
    # several lists of 1, 2 and 4 registers, in batches of 2 to 8
    (128, 32, 64, 2, "dup", 3, 1),
    (128, 32, 128, 4, "real", 3, 1),
    (96, 32, 256, 4, "dup", 1, 1),
    (128, 64, 256, 2, "real", 3, 1),
    (128, 64, 256, 4, "dup", 3, 1),
    (64, 32, 256, 8, "real", 3, 1),
    (64, 128, 128, 2, "dup", 3, 1),
    # more hashes than are computed ahead
    (128, 64, 32, 1, "real", 4, 1),
    (128, 32, 128, 4, "dup", 10, 1),
    # degree 16: two lists per register, up to 4 lists
    (128, 16, 16, 1, "dup", 3, 1),
    (128, 16, 64, 4, "real", 4, 1),
    (64, 16, 256, 4, "real", 3, 1),
    # random entries over several entry batches
    (128, 16, 256, 1, "real", 3, 0),
    (128, 32, 256, 2, "dup", 3, 0),
    # rows of any chunk count, and 30 chunks with wide batches
    (200, 64, 128, 2, "dup", 3, 1),
    (960, 64, 256, 4, "real", 3, 1),
    (960, 32, 128, 4, "dup", 3, 1),
]


def _data(d, kind, R, n, nq):
    base, q = _mixture(n, nq, d, kind == "dup", seed=11 * d + R + n)
    if kind == "dup":
        rng = np.random.Generator(np.random.Philox(d + R))
        base[n // 2:] = base[rng.integers(0, n // 2, n - n // 2)]
    return base, q


@pytest.mark.parametrize("team", [1, 8])
@pytest.mark.parametrize("d,R,L,W,kind,nh,mode", CASES)
def test_merge_and_filter_paths_match_oracle(lib, orc, cuda, d, R, L, W, kind, nh, mode, team):
    from rt_entry_gb300 import datasets as ds
    base, q = _data(d, kind, R, 1500, 120)
    graph = ds.knn_graph(base, R)
    idx = _index(base, graph, 24, 0.2)
    _, _, pids = idx.kdtree()
    kw = dict(search_width=W, bloom_hashes=nh, entry_mode=mode)
    ids, dd = idx.search_projected(q, beam=L, k=L, team_warps=team, **kw)
    oids, od, ocnt = orc.search(base, q, graph, L=L, k=L, leaf_pids=pids, hits=idx.locate(q),
                                with_counters=True, **kw)
    assert np.array_equal(ids, oids), f"{(ids != oids).any(1).sum()} queries differ"
    assert np.array_equal(dd, od)
    assert np.array_equal(idx.counters(q, beam=L, k=L, team_warps=team, **kw), ocnt[:, :4])


@pytest.mark.parametrize("d", [40, 64, 96, 100, 128, 160])
def test_bf16_copy_holds_the_rounded_base(lib, cuda, d):
    """The paired BF16 layout (2 to 4 chunks) and the plain one read back as
    the base rounded to BF16."""
    import rt_entry_gb300 as r
    base, _ = _mixture(300, 4, d, False, seed=d)
    idx = r.Index.from_arrays(base, (np.arange(300)[:, None] + np.arange(1, 17)) % 300)
    want = (r.bf16_bits(base).astype(np.uint32) << 16).view(np.float32)
    assert np.array_equal(idx.search_base_lowp(r.PREC_BF16), want)


@pytest.mark.parametrize("d,L,W", [(64, 32, 1), (96, 16, 4), (128, 32, 4), (128, 64, 1)])
def test_bf16_rows_of_two_to_four_chunks_match_oracle(lib, orc, cuda, d, L, W):
    """Rows in the paired layout, on the tensor cores and (2 chunks, or a pool
    and batch without a tensor-core kernel) in the kernels for any chunk
    count.  Integer values: every distance is exact on both."""
    import rt_entry_gb300 as r
    from rt_entry_gb300 import datasets as ds
    base, q = _mixture(1500, 100, d, True, seed=3 * d + L)
    graph = ds.knn_graph(base, 64 if W < 4 else 32)
    idx = _index(base, graph, 24, 0.2)
    _, _, pids = idx.kdtree()
    ids, dd = idx.search_projected(q, beam=L, k=L, search_width=W, precision=r.PREC_BF16)
    oids, od = orc.search(idx.search_base_lowp(r.PREC_BF16), q, graph, L=L, k=L, search_width=W, leaf_pids=pids,
                          hits=idx.locate(q))
    assert np.array_equal(ids, oids) and np.array_equal(dd, od)
