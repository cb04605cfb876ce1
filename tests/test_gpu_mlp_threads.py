"""Calls on one network from several threads run one after the other."""
import threading
import time

import numpy as np
import pytest

from nvshmem_b200 import picker as P

pytestmark = pytest.mark.gpu


def test_parameters_set_during_training():
    """Weights set while another thread trains (600 rows to a batch: a launch per
    step) take effect before the training or after it, never between steps."""
    rng = np.random.default_rng(8)
    X = rng.normal(size=(1200, 6)).astype(np.float32)
    Y, M = rng.normal(size=(1200, 12)).astype(np.float32), np.ones((1200, 12), np.float32)
    a, b = P.MLP(seed=5), P.MLP(seed=6)
    new = b.params()

    def train(net):
        net.train(X, Y, M, epochs=400, batch=600, lr=1e-3, seed=2)

    train(b)  # what training from `new` gives
    t = threading.Thread(target=train, args=(a,))
    t.start()
    time.sleep(0.02)  # the 800 steps take some 60 ms
    a.set_params(new)
    t.join()
    got = a.params()
    # float32 sums in another order, 800 steps of at most 1e-3 each
    assert np.array_equal(got, new) or np.abs(got - b.params()).max() < 0.05
    a.close()
    b.close()
