"""Loss and gradient of the proposal network (mlp_train_kernel: tiles of 32
records, partial gradients per CTA) against float64 torch autograd, at batch
sizes around a tile, a full grid of tiles and more than one tile per CTA;
and Adam steps against the same steps taken from the returned gradients.
Tolerances are those of the network's other gradient test (FP32 sums against
FP64: loss 1e-4 relative, gradient 2e-3 of its largest component).
"""
import numpy as np
import pytest

from test_gpu_learned import torch_loss

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def recorded():
    import cuda_pspin_b200 as ps
    eng = ps.Engine(ps.default_config(N=12, nrep=32, seed=9))
    _, betas = ps.temperature_schedule(8, 0.3, 1.5, True)
    eng.pt_init(8, 4, betas, 1)
    eng.learn_init(seed=4, capacity=1 << 15, record_prob=1.0)
    eng.set_proposal(ps.PROPOSAL_PLAIN_FIELDS)
    eng.pt_run(200)
    n, rec = eng.learn_records(1 << 15)
    yield eng, rec
    eng.free()


@pytest.mark.parametrize("n", [1, 31, 33, 9472, 9473, 20001])
def test_loss_and_gradient(recorded, n):
    eng, rec = recorded
    r = np.resize(rec, (n, rec.shape[1]))
    loss, g = eng.learn_loss_grad(r)
    ref, gref = torch_loss(eng.learn_params(), r)
    assert abs(loss - ref) <= 1e-4 * abs(ref)
    assert np.abs(g - gref).max() <= 2e-3 * np.abs(gref).max()


def test_training_step_is_adam(recorded):
    """One step on a ring whose every draw is the same record set: the first
    Adam step moves each weight by lr g / (|g| + eps sqrt-corrected)."""
    import cuda_pspin_b200 as ps
    eng, rec = recorded
    w0 = eng.learn_params()
    eng.learn_train(1, 64, 1e-3)
    step = eng.learn_params() - w0
    # |m / c1| = |g|, sqrt(v / c2) = |g|: a step of lr wherever |g| >> eps, never more
    assert np.abs(step).max() <= 1.001e-3 and (np.abs(step) > 0.9e-3).mean() > 0.5
