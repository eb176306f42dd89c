"""GPU checks of the warm-start network's tensor-core kernels against the FP64
oracle (oracle/mlp.py): forward, parameter gradients, Adam, and training."""
import numpy as np
import pytest

from oracle import mlp as OM
from phybs_gb300 import _lib as L
from phybs_gb300.warmstart import MLPTrainer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from phybs_gb300.build import build
    build()


def _data(n, seed=0):
    rng = np.random.default_rng(seed)
    X = rng.normal(0.0, 1.0, (n, 24)).astype(np.float32)
    Y = np.stack([np.sin(X[:, 0]) + 0.5 * X[:, 1] * X[:, 2], np.tanh(X[:, 3] - X[:, 4]), 0.3 * X[:, 5] ** 2 - 0.2],
                 axis=1).astype(np.float32)
    return X, Y


def test_param_count_matches_oracle():
    t = MLPTrainer(seed=1)
    assert t.n_params == OM.N_PARAMS == 10115
    t.close()


def test_forward_matches_oracle():
    theta = OM.init_params(3).astype(np.float32)
    t = MLPTrainer(theta)
    X, _ = _data(1000, 1)
    y = t.forward(X)
    ref, _ = OM.forward(theta, X, round_bf16=True)
    ref64, _ = OM.forward(theta, X, round_bf16=False)
    scale = np.abs(ref).max()
    assert np.abs(y - ref).max() / scale < 2e-2
    # the BF16 network against the all-FP64 one, stated as a bound
    assert np.abs(y - ref64).max() / np.abs(ref64).max() < 5e-2
    t.close()


@pytest.mark.parametrize("n", [37, 300, 4096])
def test_gradient_matches_oracle(n):
    """Every parameter block's gradient against the FP64 backward with the
    kernels' BF16 operand rounding: relative error of the block norm < 5e-3
    (measured 2.2e-3 at most, on the 37-sample batch), cosine > 0.999."""
    theta = OM.init_params(5).astype(np.float32)
    t = MLPTrainer(theta)
    X, Y = _data(n, 2)
    loss, g = t.gradient(X, Y)
    lref, gref = OM.loss_and_grad(theta, X, Y, round_bf16=True)
    assert abs(loss - lref) / lref < 1e-2
    off = 0
    errs = []
    for o, i in OM.SIZES:
        for sz in (o * i, o):
            a, b = g[off:off + sz].astype(np.float64), gref[off:off + sz]
            off += sz
            nb = np.linalg.norm(b)
            errs.append(np.linalg.norm(a - b) / nb)
            assert np.linalg.norm(a - b) / nb < 5e-3, (off, np.linalg.norm(a - b) / nb)
            assert a @ b / (np.linalg.norm(a) * nb) > 0.999
    print(f"n={n}: per-block gradient error {[f'{e:.1e}' for e in errs]}")
    t.close()


def test_adam_step_matches_oracle():
    theta = OM.init_params(7).astype(np.float32)
    t = MLPTrainer(theta)
    X, Y = _data(512, 3)
    _, g = t.gradient(X, Y)
    t.set_data(X, Y)
    t.train(1, batch=512, lr=1e-3, seed=0)
    new = t.params.astype(np.float64)
    ref, _, _ = OM.adam(theta.astype(np.float64), np.zeros_like(new), np.zeros_like(new), g.astype(np.float64), 1, 1e-3)
    assert np.abs(new - ref).max() < 1e-6 + 1e-5 * np.abs(ref).max()
    t.close()


def test_weighted_adam_step_matches_oracle():
    """With per-sample loss weights, one full-batch Adam step moves every
    parameter by -lr * sign of the FP64 weighted gradient (Adam's first step),
    wherever that gradient is clearly non-zero."""
    theta = OM.init_params(9).astype(np.float32)
    t = MLPTrainer(theta)
    X, Y = _data(512, 5)
    W = np.random.default_rng(6).uniform(0.0, 4.0, 512).astype(np.float32)
    t.set_data(X, Y, W)
    lr = 1e-3
    t.train(1, batch=512, lr=lr, seed=0)
    step = t.params.astype(np.float64) - theta
    _, g = OM.loss_and_grad(theta, X, Y, round_bf16=True, W=W)
    clear = np.abs(g) > 1e-2 * np.abs(g).max()
    assert clear.sum() > 1000
    np.testing.assert_allclose(step[clear], -lr * np.sign(g[clear]), rtol=1e-2, atol=1e-6)
    _, g_unw = OM.loss_and_grad(theta, X, Y, round_bf16=True)
    assert (np.sign(g_unw[clear]) != np.sign(g[clear])).any()  # the weights changed the step
    t.close()


def test_training_reduces_loss():
    t = MLPTrainer(seed=11)
    X, Y = _data(20000, 4)
    t.set_data(X, Y)
    losses = t.train(400, batch=1024, lr=2e-3, seed=1)
    assert losses[-20:].mean() < 0.25 * losses[:5].mean(), (losses[:5], losses[-20:])
    t.close()


# rows about the tile and grid lines: 1; a 16-row fragment's edge; one tile and
# one row more; two steps a launch's limit apart; one tile a SM and one more
# (152 x 64 = 9,728)
@pytest.mark.parametrize("n,steps", [(1, 2), (17, 3), (64, 3), (65, 3), (300, 66), (9728, 2), (9729, 2)])
@pytest.mark.parametrize("weighted", [False, True])
def test_steps_of_one_launch_match_adam(n, steps, weighted):
    """Steps on the whole set as one minibatch against FP64 Adam on the
    gradients of the same parameters (weights of 2: twice the gradient).  The
    bound: an FP32 update's rounding, and a gradient's (1e-5 of an update of at
    most lr) where rows are summed in another order, a step."""
    theta = OM.init_params(11).astype(np.float32)
    X, Y = _data(n, 4)
    a, b = MLPTrainer(theta), MLPTrainer(theta)
    a.set_data(X, Y, np.full(n, 2.0, np.float32) if weighted else None)
    b.set_data(X, Y)
    ref, m, v = theta.astype(np.float64), np.zeros(a.n_params), np.zeros(a.n_params)
    losses = a.train(steps, batch=n, lr=1e-3, seed=0)
    scale = 2.0 if weighted else 1.0
    if steps > 4:  # too long for the gradients' sensitivity: one launch against two
        got = a.params
        b.set_data(X, Y, np.full(n, 2.0, np.float32) if weighted else None)
        lb = b.train(steps, batch=n, lr=1e-3, seed=0)
        assert np.array_equal(got, b.params) and np.array_equal(losses, lb)
        assert np.all(np.isfinite(losses)) and losses[-1] < losses[0]
    else:
        for k in range(steps):
            b.params = ref.astype(np.float32)
            loss, g = b.gradient(X, Y)
            assert abs(losses[k] - scale * loss) <= 1e-4 * scale * loss
            ref, m, v = OM.adam(ref, m, v, scale * g.astype(np.float64), k + 1, 1e-3)
        assert np.abs(a.params - ref).max() < steps * (1e-6 + 1e-5 * np.abs(ref).max())
    a.close()
    b.close()


# (rows, batch, steps): batches below a tile, not a multiple of it, beyond one
# tile a SM; several epochs, rows left over in each; more steps an epoch than a
# launch takes (64), once with rows left over
@pytest.mark.parametrize("n,batch,steps", [(1000, 16, 130), (1000, 99, 25), (4097, 64, 70), (5000, 333, 31),
                                           (30001, 9729, 7), (65, 64, 5)])
@pytest.mark.parametrize("weighted", [False, True])
def test_steps_of_one_launch_equal_single_steps(n, batch, steps, weighted):
    """Minibatches of one launch (rows found on the device, weights carried from
    step to step there) against the same ones a launch each: bit for bit."""
    theta = OM.init_params(5).astype(np.float32)
    X, Y = _data(n, 6)
    W = np.random.default_rng(7).uniform(0.2, 3.0, n).astype(np.float32) if weighted else None
    out = []
    for cap in (64, 1):
        t = MLPTrainer(theta)
        assert L.lib().pbs_mlp_test_launch_steps(t._t, cap) == 0
        t.set_data(X, Y, W)
        out.append((t.train(steps, batch=batch, lr=1e-3, seed=9), t.params))
        t.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert not np.array_equal(out[0][1], theta)


@pytest.mark.parametrize("n,batch", [(6400, 100), (9600, 96), (4096, 1024)])
def test_an_epoch_takes_every_row_once(n, batch):
    """With a step too small to change a parameter (1e-30; the biases start at 0
    and stay below what a sum notices) the mean loss of an epoch's minibatches
    is the loss of all rows.  Both are FP32 sums of n
    positive terms: they agree to a few times 2^-24 sqrt(n), below 1e-5."""
    theta = OM.init_params(5).astype(np.float32)
    X, Y = _data(n, 8)
    Y *= np.linspace(0.1, 3, n, dtype=np.float32)[:, None]  # no two rows weigh the same
    t = MLPTrainer(theta)
    full, _ = t.gradient(X, Y)
    t.set_data(X, Y)
    losses = t.train(n // batch, batch=batch, lr=1e-30, seed=3)
    assert np.array_equal(t.params[theta != 0], theta[theta != 0])
    assert abs(losses.astype(np.float64).mean() - full) <= 1e-5 * full
    t.close()


def test_failed_launch_takes_no_adam_step():
    """Training after a launch that failed is training from where it was: the
    step count of Adam's bias correction goes on from the steps taken."""
    X, Y = _data(500, 3)
    out = []
    for fail in (False, True):
        t = MLPTrainer(seed=4)
        t.set_data(X, Y)
        t.train(3, batch=100, seed=0)
        if fail:
            assert L.lib().pbs_mlp_test_refuse(t._t) == 0
            with pytest.raises(L.PhybsError):
                t.train(4, batch=100, seed=1)
        out.append((t.train(2, batch=100, seed=2), t.params))
        t.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
