"""Host threads that share a model get the rows of single calls."""
import threading

import numpy as np
import pytest

from sph_gb300 import LearnedModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1000, 777), (20000, 130), (131073, 40000)])
def test_forward_from_two_threads(cuda_lib, sizes):
    rng = np.random.default_rng(sum(sizes))
    rows = [rng.standard_normal((n, LearnedModel.IN)).astype(np.float32) for n in sizes]
    with LearnedModel(0, seed=4) as m:
        ref = [m.forward(x) for x in rows]
    with LearnedModel(0, seed=4) as m:  # its workspace is made by the threads
        bad = []

        def calls(k):
            for _ in range(20):
                if not np.array_equal(m.forward(rows[k]), ref[k]):
                    bad.append(k)

        threads = [threading.Thread(target=calls, args=(k,)) for k in (0, 1)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not bad
