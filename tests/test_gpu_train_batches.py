"""The training kernels at the edges of their 16-sample blocks, 32-sample
stages and batch slices (64 samples and up, at most 24), against the FP64
restatement; repeated calls give the same bits."""
import numpy as np
import pytest

import __graft_entry__ as g
import systems as S

nbg = S.nbg
learned = g.load_learned_oracle()
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(gpu):
    sim, pos, vel, L = S.spcfw_water_rf(1000, thermo=False)
    desc, keep = nbg.system_descriptor(sim)
    eng = nbg.Engine(desc, 0)
    eng.ml_enable()
    eng.ml_init_params(seed=3, w1_scale=1.0)
    return eng


# FP32 forward and backward (128-term sums) and sums over the batch: 1e-5 of the gradient's norm
@pytest.mark.parametrize("species", [0, 1])
@pytest.mark.parametrize("B", [1, 15, 17, 63, 65, 129, 1536, 1537, 3001])
def test_batch_gradient(engine, species, B):
    rng = np.random.default_rng(B)
    x = rng.standard_normal((B, 64)).astype(np.float32)
    y = rng.standard_normal(B).astype(np.float32)
    loss, grad = engine.ml_batch_gradient(species, x, y)
    _, ref = learned.train_gradients(engine.ml_get_params(species).astype(np.float64), x.astype(np.float64),
                                            y.astype(np.float64))
    assert np.linalg.norm(grad - ref) <= 1e-5 * np.linalg.norm(ref)
    again = engine.ml_batch_gradient(species, x, y)
    assert again[0] == loss and np.array_equal(again[1], grad)
