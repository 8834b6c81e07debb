"""The automatic choice of warps per query on both sides of each of its lines,
on the host for rte_search and on the device for the batcher's graph: the
number chosen, and results equal to those of one warp per query."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _index(d, R, n=1500, seed=3):
    import rt_entry_gb300 as r
    rng = np.random.Generator(np.random.Philox(seed + d + R))
    cent = 100 * rng.random((12, d))
    base = (cent[rng.integers(0, 12, n)] + 5 * rng.standard_normal((n, d))).astype(np.float32)
    ring = ((np.arange(n)[:, None] + np.arange(1, R + 1)) % n).astype(np.int32)
    return r.Index.from_arrays(base, ring).build_kdtree(24, 0.2), base, rng


# d, degree, precision, beam, width, [(batch in resident warps, warps per query up to it)]; one above
LINES = [
    (128, 64, 0, 32, 1, [(10, 2)]),
    (128, 64, 0, 128, 1, [(3, 2)]),
    (64, 32, 0, 128, 1, []),
    (128, 64, 0, 256, 1, []),
    (128, 64, 1, 32, 1, [(2, 2)]),
    (128, 32, 1, 16, 1, [(1, 1), (2, 2)]),
    (64, 32, 1, 32, 2, [(1, 1), (2, 2)]),
    (128, 64, 1, 128, 1, []),
    (96, 32, 2, 32, 1, [(10, 2)]),
    (128, 32, 2, 32, 1, []),
    (128, 16, 0, 32, 1, [(1, 1), (2, 2)]),
    (128, 16, 0, 128, 1, []),
    (128, 16, 1, 32, 1, [(1, 1), (2, 2)]),
    (256, 16, 1, 64, 1, [(1, 1), (2, 2)]),
    (128, 16, 2, 64, 1, []),
    (256, 32, 0, 16, 1, [(3, 2)]),
    (256, 32, 0, 64, 1, [(10, 2)]),
    (256, 32, 1, 64, 1, [(2, 2)]),
    (256, 32, 2, 64, 1, []),
    (960, 64, 0, 64, 1, [(2, 4), (10, 2)]),
    (960, 64, 0, 256, 4, [(2, 4), (10, 2)]),
    (960, 64, 1, 64, 1, [(2, 4), (5, 2)]),
    (960, 64, 2, 256, 1, [(1, 4)]),
    (960, 64, 2, 256, 4, [(2, 4)]),
]


@pytest.mark.parametrize("d,R,prec,L,W,lines", LINES)
def test_the_choice_on_both_sides_of_each_line(lib, cuda, d, R, prec, L, W, lines):
    idx, _, _ = _index(d, R)
    kw = dict(beam=L, k=10, search_width=W, precision=prec)
    _, res = idx.search_team(1, **kw)
    assert res >= 1024
    below = res // 2 + 1  # above it a batch leaves no warps over
    for load, warps in lines:
        assert idx.search_team(below, **kw)[0] == warps
        assert idx.search_team(load * res, **kw)[0] == warps, (load, warps)
        below = load * res + 1
    assert idx.search_team(below, **kw)[0] == 1
    assert idx.search_team(200 * res, **kw)[0] == 1
    assert idx.search_team(res // 8, **kw)[0] == 8  # small batches: every warp
    assert idx.search_team(200 * res, team_warps=8, **kw)[0] == 8


def test_rows_beyond_l2_take_two_warps(lib, cuda):
    """2.9M x 96: 557 MB of BF16 rows and 278 MB of FP8 rows, above their lines."""
    import torch

    import rt_entry_gb300 as r
    n = 2_900_000
    ring = (torch.arange(n, device="cuda", dtype=torch.int32)[:, None]
            + torch.arange(1, 33, device="cuda", dtype=torch.int32)) % n
    idx = r.Index.from_arrays(torch.zeros((n, 96), device="cuda"), ring)
    for prec, L, W, lines in [(1, 64, 1, [(10, 2)]), (1, 128, 2, [(10, 2)]), (1, 16, 1, [(1, 1), (10, 2)]),
                              (1, 256, 4, [(3, 2)]), (2, 128, 1, [(2, 2)]), (2, 256, 1, []), (0, 256, 1, [])]:
        kw = dict(beam=L, k=10, search_width=W, precision=prec, entry_mode=r.ENTRY_RANDOM)
        _, res = idx.search_team(1, **kw)
        below = res // 2 + 1
        for load, warps in lines:
            assert idx.search_team(below, **kw)[0] == warps, (prec, L)
            assert idx.search_team(load * res, **kw)[0] == warps, (prec, L)
            below = load * res + 1
        assert idx.search_team(below, **kw)[0] == 1, (prec, L)


@pytest.mark.parametrize("d,R,prec,L,loads", [
    (64, 64, 0, 16, (10,)),          # two warps, then one
    (128, 32, 1, 16, (1, 2)),        # one, two, one
    (960, 64, 1, 16, (2, 5)),        # four, two, one
])
def test_batches_past_each_line_give_the_single_warps_results(lib, cuda, d, R, prec, L, loads):
    import rt_entry_gb300 as r
    idx, base, rng = _index(d, R)
    kw = dict(beam=L, k=10, precision=prec, max_iter=6)
    _, res = idx.search_team(1, **kw)
    cap = loads[-1] * res + 1
    q = base[rng.integers(0, len(base), cap)] + rng.standard_normal((cap, d)).astype(np.float32)
    want, wd = idx.search(q, params=r.default_params(team_warps=1, **kw))
    p = r.default_params(**kw)
    b = idx.batcher(cap, params=p)
    for m in {m for load in loads for m in (load * res, load * res + 1)} | {37}:
        for got, gd in (idx.search(q[:m], params=p), b.search(q[:m])):
            assert np.array_equal(got, want[:m]) and np.array_equal(gd, wd[:m]), m
    b.close()
