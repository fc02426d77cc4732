"""Inference of one learner from several threads: calls share its input and output buffers, each
gets its own samples' outputs."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tensor_cores", [True, False])
def test_infer_from_threads(ccx, tensor_cores):
    r = np.random.RandomState(7)
    m = ccx.Learner()
    # sizes that grow, so that the buffers are replaced while other threads call
    X = [r.standard_normal((n, 18)).astype(np.float32) for n in (100, 1000, 9000, 30000)]
    want = [m.infer(x, tensor_cores=tensor_cores) for x in X[::-1]][::-1]
    m2 = ccx.Learner()
    m2.infer(X[0][:1], tensor_cores=tensor_cores)
    got, bar = [[] for _ in X], threading.Barrier(len(X))

    def work(i):
        bar.wait()
        for _ in range(20):
            got[i].append(m2.infer(X[i], tensor_cores=tensor_cores))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(X))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for w, g in zip(want, got):
        assert len(g) == 20 and all(np.array_equal(w, x) for x in g)
