"""The kNN builder's thresholded pass at its edges, against an FP64 brute
force on the host: tile remainders (128 rows, 256 columns), the smallest base
it takes, resident and streamed operand blocks (d up to 128, above), rows that
it leaves to the stored products (duplicates, degrees above 128), and unsorted
and cluster-sorted bases."""
import numpy as np
import pytest

from test_gpu_knn import _mixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,R,integer", [
    (1023, 40, 16, True),     # below the pass's smallest base
    (1024, 40, 16, True),     # the smallest
    (1025, 33, 1, False),     # one row and one column past a tile, degree 1
    (2177, 128, 64, True),
    (3333, 129, 32, False),   # operands streamed, rows of odd length
    (2600, 130, 128, True),   # the largest degree
    (2600, 64, 129, True),    # above it
    (17000, 24, 32, False),   # two row blocks
])
def test_filtered_graph_matches_fp64_brute_force(lib, cuda, n, d, R, integer):
    import rt_entry_gb300 as r
    from rt_entry_gb300 import datasets as ds
    base = _mixture(n, d, integer, seed=n + d + R)
    assert np.array_equal(r.knn_graph(base, R), ds.knn_graph(base, R, device="cpu"))


def test_cluster_sorted_base_and_repeated_rows(lib, cuda):
    """Rows in cluster order (a thread's columns hold all of a row's
    neighbours or none), and one row repeated more often than the candidates
    of a row that the pass can finish (the stored products take up to 1024)."""
    import rt_entry_gb300 as r
    from rt_entry_gb300 import datasets as ds
    base = _mixture(6000, 64, True, seed=5)
    base = base[np.lexsort(base.T[:3])]
    base[2000:2700] = base[2000]
    assert np.array_equal(r.knn_graph(base, 32), ds.knn_graph(base, 32, device="cpu"))
