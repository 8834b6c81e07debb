"""The training step on three streams against the same step on one, and the
labels that training makes on the device, bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = lambda a: a.ctypes.data_as(ctypes.c_void_p)


def _steps(lib, side, X, y, Ws, lr):
    import rt_entry_gb300 as r
    steps, M, d = X.shape
    H, C = Ws[0].shape[0], Ws[4].shape[0]
    n = sum(w.size for w in Ws)
    grads, weights, loss = np.empty((steps, n), np.float32), np.empty(n, np.float32), np.empty((steps, M), np.float32)
    ptrs = (ctypes.c_void_p * 6)(*[w.ctypes.data for w in Ws])
    r._check(lib.rte_mlp_steps_check(P(X), P(y), steps, M, d, H, C, ptrs, lr, side, P(grads), P(weights), P(loss)))
    return grads, weights, loss


@pytest.mark.parametrize("M,d,H,C", [(128, 8, 8, 8), (1024, 96, 256, 1000), (4096, 128, 256, 4096), (256, 40, 512, 64)])
def test_side_streams_give_the_same_bits(lib, cuda, M, d, H, C):
    """Six steps without a host wait and with large updates: a transpose of an
    earlier step's weights or activations would change every later gradient."""
    rng = np.random.Generator(np.random.Philox(M + d + H + C))
    steps = 6
    X = rng.standard_normal((steps, M, d)).astype(np.float32)
    y = rng.integers(0, C, (steps, M)).astype(np.int32)
    Ws = []
    for o, i in ((H, d), (H, H), (C, H)):
        Ws += [(rng.standard_normal((o, i)) * np.sqrt(2.0 / i)).astype(np.float32),
               (0.1 * rng.standard_normal(o)).astype(np.float32)]
    want = _steps(lib, 0, X, y, Ws, 0.05)
    assert np.isfinite(want[0]).all()
    assert all((want[0][t] != want[0][t + 1]).any() for t in range(steps - 1))
    for _ in range(3):
        got = _steps(lib, 1, X, y, Ws, 0.05)
        for a, b in zip(got, want):
            assert a.tobytes() == b.tobytes()


def test_training_twice_gives_one_entry(lib, cuda):
    import rt_entry_gb300 as r
    from rt_entry_gb300 import datasets as ds
    mix = ds.mixture_config(2)
    base = mix.sample(10000, ds.SEED_BASE)
    idx = r.Index.from_arrays(base, ds.knn_graph(base, 32)).build_pca().build_kdtree(32, 0.2)
    q = mix.sample(20000, ds.SEED_TRAIN)
    probe = idx.project(mix.sample(3000, ds.SEED_QUERY))
    runs = []
    for _ in range(2):
        rep = idx.train_learned(q, hidden=128, epochs=2, batch=2048, max_classes=256)
        runs.append((rep["first_loss"], rep["last_loss"], rep["train_acc"], idx.learned_leaves(probe)))
    assert runs[0][:3] == runs[1][:3]
    assert np.array_equal(runs[0][3], runs[1][3])


@pytest.mark.parametrize("np_,leaves,cap", [(1, 1, 1), (1000, 50, 24), (4097, 257, 16)])
def test_labels_match_the_host_loop(lib, cuda, np_, leaves, cap):
    import rt_entry_gb300 as r
    rng = np.random.Generator(np.random.Philox(np_))
    pids = np.full((leaves, cap), np_, np.int32)  # padding
    order = rng.permutation(np_)
    listed = order[: min(np_, leaves * cap * 3 // 4 + 1)]  # the rest is in no leaf
    slots = rng.choice(leaves * cap, len(listed), replace=False)
    pids.reshape(-1)[slots] = listed
    pids[0, -1] = max(pids[0, -1], np_)  # a leaf with padding
    cls = rng.integers(0, 9, leaves).astype(np.int32)
    ids = np.concatenate([rng.integers(0, np_, 500), [-1, np_, np_ - 1, 0, 2**31 - 1]]).astype(np.int32)
    leaf_of = np.zeros(np_, np.int64)
    for l in range(leaves):
        for p in pids[l]:
            if p < np_:
                leaf_of[p] = l
    want = np.array([cls[leaf_of[i]] if 0 <= i < np_ else cls[0] for i in ids], np.int32)
    got = np.empty_like(ids)
    r._check(lib.rte_point_labels_check(P(ids), len(ids), P(pids), leaves, cap, np_, P(cls), P(got)))
    assert np.array_equal(got, want)
