"""Where the batcher's results go: straight to device memory and page-locked
host memory, by copies to pageable memory and to page-locked memory that a
4-byte store cannot address."""
import numpy as np
import pytest

from test_gpu_stream import _index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 10, 64])
def test_batcher_outputs_of_every_kind(lib, cuda, k):
    import torch

    import rt_entry_gb300 as r
    idx, base, q = _index(nq=700)
    p = r.default_params(beam=64, k=k)
    want, wd = idx.search(q, params=p)
    b = idx.batcher(700, params=p)
    pinned = torch.from_numpy(q).pin_memory()
    for s, e in [(0, 700), (3, 4), (10, 143)]:
        m = e - s
        ids = torch.empty((m, k), dtype=torch.int32).pin_memory()
        dd = torch.empty((m, k), dtype=torch.float32).pin_memory()
        dev_ids = torch.empty((m, k), dtype=torch.int32, device="cuda")
        # page-locked, 2 bytes past a 4-byte boundary
        raw = torch.zeros(8 * m * k + 16, dtype=torch.uint8).pin_memory().numpy()
        odd_ids = np.ndarray((m, k), "<i4", raw.data, 2)
        odd_dd = np.ndarray((m, k), "<f4", raw.data, 4 * m * k + 6)
        page_ids, page_dd = np.empty((m, k), np.int32), np.empty((m, k), np.float32)
        for out_ids, out_dd in ((ids, dd), (dev_ids, dd), (ids, page_dd), (page_ids, page_dd)):
            b.search(pinned[s:e], out_ids=out_ids, out_dists=out_dd)
            got = out_ids.cpu().numpy() if torch.is_tensor(out_ids) else out_ids
            gd = out_dd.numpy() if torch.is_tensor(out_dd) else out_dd
            assert np.array_equal(got, want[s:e]) and np.array_equal(gd, wd[s:e]), (s, e)
            ids.zero_(), dd.zero_(), dev_ids.zero_(), page_ids.fill(0), page_dd.fill(0)
        r._check(r.load_library().rte_batcher_search(b._h, pinned[s:e].data_ptr(), m, odd_ids.ctypes.data,
                                                     odd_dd.ctypes.data, None))
        assert np.array_equal(odd_ids, want[s:e]) and np.array_equal(odd_dd, wd[s:e])
        r._check(r.load_library().rte_batcher_search(b._h, pinned[s:e].data_ptr(), m, ids.data_ptr(), None, None))
        assert np.array_equal(ids.numpy(), want[s:e])  # no distances asked for
    b.close()
