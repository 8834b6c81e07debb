"""Batches up to 4096 queries launch their chain of kernels programmatically,
larger ones plainly: both sides of the line, and many calls in flight on one
stream at once, give every query what one plainly launched batch gives it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ["kdtree", "learned"])
@pytest.mark.parametrize("team", [0, 1])
def test_chained_launches_equal_one_plain_batch(lib, cuda, entry, team):
    import torch

    import rt_entry_gb300 as r
    from rt_entry_gb300 import datasets as ds
    mix = ds.mixture_config(2)
    base = mix.sample(20000, ds.SEED_BASE)
    q = mix.sample(4700, ds.SEED_QUERY)
    idx = r.Index.from_arrays(base, ds.knn_graph(base, 32)).build_pca().build_kdtree(32, 0.2)
    kw = dict(beam=32, k=10)
    if entry == "learned":
        idx.train_learned(mix.sample(4096, ds.SEED_TRAIN), hidden=128, epochs=1, batch=2048, label_beam=32,
                          max_classes=64)
        kw.update(entry_mode=r.ENTRY_LEARNED, precision=1, rerank=1)
    want, wd = idx.search(q, params=r.default_params(team_warps=1, **kw))
    p = r.default_params(team_warps=team, **kw)
    qt = torch.from_numpy(q).cuda()
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    cuts = [(0, 4096), (0, 4097), (500, 4595), (4699, 4700), (0, 1), (7, 40), (1, 300)] * 3
    outs = []
    with torch.cuda.stream(st):
        for s, e in cuts:  # no synchronisation in between
            part = qt[s:e].contiguous()
            outs.append((idx.search(part, params=p, stream=st), part))
    st.synchronize()
    for (s, e), ((ids, dd), _) in zip(cuts, outs):
        assert np.array_equal(ids.cpu().numpy(), want[s:e]) and np.array_equal(dd.cpu().numpy(), wd[s:e]), (s, e)
