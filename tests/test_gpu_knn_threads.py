"""Graph builds of different degrees at once, each from its own thread: the
block sizes of one build must not change the launch limits of another's."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_builds_of_two_degrees_at_once(lib, cuda):
    import torch

    import rt_entry_gb300 as r
    rng = np.random.Generator(np.random.Philox(4))
    base = torch.from_numpy(rng.standard_normal((1500, 16)).astype(np.float32)).cuda()
    want = {R: r.knn_graph(base, R).cpu() for R in (16, 128)}
    errors = []

    def work(R):
        try:
            for _ in range(300):
                if not torch.equal(r.knn_graph(base, R).cpu(), want[R]):
                    errors.append(f"degree {R}: another graph")
        except Exception as e:  # noqa: BLE001
            errors.append(f"degree {R}: {e}")

    threads = [threading.Thread(target=work, args=(R,)) for R in (16, 128, 16)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]
