"""The network's gradients at sizes where a block takes several tiles or a part of
one: the training kernel has at most 148 blocks with tiles of up to 64 samples.

Tolerance: that of the comparison at 777 samples. The sum over samples grows as its
rounding does for targets of random sign, so the relative error does not depend on
their number."""
import numpy as np
import pytest

import oracle
from test_gpu_learned import GRAD_RTOL, cuda, random_net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 64, 592, 593, 9472, 9473, 16384, 18945, 40001])
def test_gradients_over_tiles(n):
    m, p = random_net(6)
    rng = np.random.default_rng(n)
    f = rng.standard_normal((n, 24)).astype(np.float32)
    t = rng.standard_normal((n, 3)).astype(np.float32)
    gr, lr = oracle.mlp_gradients(p, f, t)
    for _ in range(2):
        g, loss = m.gradients(cuda(f), cuda(t))
        assert abs(loss - lr) <= 1e-5 * lr
        assert np.linalg.norm(g - gr) <= GRAD_RTOL * np.linalg.norm(gr)


def test_training_step_over_tiles():
    """One Adam step on a full batch of shuffled samples: the same gradient through the index."""
    n, lr = 18945, 1e-3
    m, p = random_net(6)
    rng = np.random.default_rng(2)
    f = rng.standard_normal((n, 24)).astype(np.float32)
    t = rng.standard_normal((n, 3)).astype(np.float32)
    g, _ = oracle.mlp_gradients(p, f, t)
    m.train(cuda(f), cuda(t), batch=n, steps=1, lr=lr, seed=0)
    clear = np.abs(g) > 1e-3 * np.abs(g).max()  # elsewhere the step's sign is the rounding's
    assert np.abs(m.parameters() - (p - lr * np.sign(g)))[clear].max() <= 1e-6 + 1e-3 * lr
