"""The sizes of the kNN builder's thresholded pass over the whole range of
bases: the lists hold what the thresholds let through, with room for the
sample's spread, and every buffer stays within bounds."""
import math

import pytest

SIZES = sorted({int(round(1024 * 1.31 ** i)) for i in range(48)} | {1023, 1024, 1572863, 1572865, 5_000_000,
                                                                   10_000_000, 12_582_912, 12_582_913, 60_000_000})


@pytest.mark.parametrize("degree", [1, 16, 32, 33, 64, 65, 128, 129, 256])
def test_lists_hold_what_the_thresholds_let_through(lib, degree):
    import rt_entry_gb300 as r
    for n in SIZES:
        p = r.knn_graph_plan(n, degree)
        if not p["thresholded"]:
            assert n < 1024 or degree > 128 or n > 80_000_000, (n, degree, p)
            continue
        # the kept count: rank n / sample on average, within a relative
        # 1 / sqrt(rank); three spreads leave one row in a thousand over
        kept = n / p["sample"] * (p["rank"] + 3.0 * math.sqrt(p["rank"]))
        assert kept <= p["cap"], (n, degree, p)
        # at least twice the degree on average, so that a threshold is rarely
        # below a row's R-th distance
        assert n / p["sample"] * (p["rank"] - 1) >= 2 * degree, (n, degree, p)
        assert p["rank"] <= 256 and p["sample"] <= n  # the threshold kernel holds 256 per row
        assert p["smem"] <= 227 * 1024
        assert p["block"] * p["sample"] * 4 <= 9 << 30 and p["block"] * p["cap"] * 8 <= 1 << 30
        assert p["block"] <= n


def test_bad_plan_arguments(lib):
    import rt_entry_gb300 as r
    for n, degree in ((0, 1), (10, 10), (1000, 0), (1000, 257), (2**31, 32)):
        with pytest.raises(r.RteError):
            r.knn_graph_plan(n, degree)
