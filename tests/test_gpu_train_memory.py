"""Device memory while a learned entry is trained: the raw queries are gone once
projected, the projected ones once they are the model's inputs."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_training_queries_are_not_held(lib, cuda):
    import torch

    import rt_entry_gb300 as r
    from rt_entry_gb300 import datasets as ds
    n, d = 1_500_000, 128
    mix = ds.mixture_config(2)
    base = mix.sample(5000, ds.SEED_BASE)
    idx = r.Index.from_arrays(base, ds.knn_graph(base, 32)).build_pca().build_kdtree(32, 0.2)
    g = torch.Generator(device="cuda").manual_seed(1)
    q = torch.from_numpy(base).cuda()[torch.randint(5000, (n,), generator=g, device="cuda")]
    q = q.cpu().numpy()  # host queries: no device copy but the library's own
    kw = dict(hidden=64, epochs=1, batch=8192, label_beam=16, max_classes=16)
    idx.train_learned(q[:16384], **kw)  # the scratch pool and modules are there
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    low, stop = [free0], threading.Event()

    def poll():
        while not stop.is_set():
            low[0] = min(low[0], torch.cuda.mem_get_info()[0])

    t = threading.Thread(target=poll)
    t.start()
    try:
        idx.train_learned(q, **kw)
    finally:
        stop.set()
        t.join()
    # queries and their projections at first, 8 n d bytes; then projections,
    # inputs (2 n d) and 16 bytes a row.  Steps, scratch and rounding are small
    # at these sizes.  Holding everything takes 10 n d + 16 n.
    peak = free0 - low[0]
    assert peak <= 8 * n * d + 16 * n + (64 << 20), f"{peak / 2**20:.0f} MiB"
