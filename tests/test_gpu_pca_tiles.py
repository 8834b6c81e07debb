"""The covariance's triangular tiles (16 x 32) and the mean's unrolled sums at
their edges: dimensions around the tile sizes, row counts around the chunk and
look-ahead sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(2, 3), (17, 15), (33, 16), (100, 17), (1023, 31), (1025, 33), (5000, 48),
                                 (8191, 65), (9000, 130)])
def test_pca_matches_fp64_on_tile_edges(lib, cuda, n, d):
    import rt_entry_gb300 as r
    rng = np.random.Generator(np.random.Philox(n + d))
    # distinct variances keep the eigenvectors well separated
    x = (rng.standard_normal((n, d)) * np.linspace(1.0, 4.0, d) + rng.uniform(-50, 50, d)).astype(np.float32)
    x[::7, 0] = 0.0
    idx = r.Index.from_arrays(x, (np.arange(n)[:, None] + np.arange(1, 17)) % n).build_pca()
    mean, rot, ev = idx.pca()
    x64 = x.astype(np.float64)
    mu = x64.mean(0)
    cov = (x64 - mu).T @ (x64 - mu) / (n - 1)
    # the mean is rounded to FP32; eigenvalues carry FP64 rounding of n terms,
    # relative to the largest
    assert np.allclose(mean, mu, rtol=2e-7, atol=1e-6)
    w = np.sort(np.linalg.eigvalsh(cov))[::-1]
    assert np.abs(ev - w).max() <= 1e-12 * max(n, d) * w[0]
    # V diagonalises the covariance to the FP32 rounding of V
    off = rot.astype(np.float64).T @ cov @ rot.astype(np.float64)
    assert np.abs(off - np.diag(ev)).max() <= 4e-7 * d * w[0]
