"""Edges of the training step's kernels, through one forward and backward pass
against the FP64 restatement: transposes and column sums with remainders of
their 64-wide tiles, softmax rows held in 4, 8 and 16 registers a thread and
read in passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,d,H,C", [
    (8, 3, 8, 5),            # below every tile
    (136, 40, 72, 200),      # remainders in every tile
    (128, 33, 64, 2048),     # 4 registers, full
    (128, 32, 64, 2049),     # 8 registers
    (128, 32, 64, 4100),     # 16 registers
    (64, 16, 16, 8200),      # passes
])
def test_step_gradients_match_fp64_restatement(lib, cuda, M, d, H, C):
    import rt_entry_gb300 as r
    from oracle import mlp_ref
    rng = np.random.Generator(np.random.Philox(M + d + C))
    X = rng.standard_normal((M, d)).astype(np.float32)
    y = rng.integers(0, C, M).astype(np.int32)
    Ws = [(rng.standard_normal(s) * np.sqrt(2.0 / s[1])).astype(np.float32) for s in ((H, d), (H, H), (C, H))]
    bs = [(0.1 * rng.standard_normal(n)).astype(np.float32) for n in (H, H, C)]
    got, loss = r.mlp_grad_check(X, y, Ws[0], bs[0], Ws[1], bs[1], Ws[2], bs[2])
    wloss, want = mlp_ref.loss_and_grads(X, y, Ws[0], bs[0], Ws[1], bs[1], Ws[2], bs[2])
    # the tolerances of the step's own test: BF16 roundings of intermediates
    # may flip where FP32 and FP64 sums differ
    assert np.allclose(loss, wloss, rtol=2e-3, atol=2e-3)
    for k, v in want.items():
        err = np.linalg.norm(got[k] - v) / max(np.linalg.norm(v), 1e-12)
        assert err < 1e-2, (k, err)
