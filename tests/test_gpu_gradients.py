"""k_gradients / k_reduce_gradients at the edges of their tiles (32 rows, at
most 296 CTAs): one batch size on each side of a tile, of the reduction's
slices and of the grid, against the oracle; and the stored-feature form that
training uses against the form that reads the states."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 31, 32, 33, 255, 257, 296 * 32, 296 * 32 + 1, 20000])
def test_gradients_at_tile_edges(batch):
    """Bound per parameter block: the 2e-3 of the network's fast exponentials
    and logarithms against float64 (test_gradients_match_oracle), which sums
    over rows keep: relative to the block's root-sum-square of |row terms| the
    row sums of 32 + 296 FP32 additions add at most 330 eps = 4e-5."""
    import mlp_oracle as mo
    from cueva.learned import LearnedSeed, synthetic_pairs
    cons, prims = synthetic_pairs(batch, seed=100 + batch)
    fit = synthetic_pairs(4096, seed=1)
    net = LearnedSeed(seed=3)
    net.fit_normalisation(*fit)
    g, loss = net.gradients(cons, prims)
    params = net.params()
    loss_ref, ref = mo.forward_backward(params[:mo.NPARAM], params[mo.NPARAM:].astype(np.float64),
                                        cons.cpu().numpy(), prims[1].cpu().numpy())
    assert abs(loss - loss_ref) <= 1e-4 * abs(loss_ref) + 1e-12
    for name, (o, n) in mo.OFF.items():
        a, b = g[o:o + n].astype(np.float64), ref[o:o + n]
        assert np.linalg.norm(a - b) <= 2.1e-3 * np.linalg.norm(b) + 1e-12, name
    g2, loss2 = net.gradients(cons, prims)
    assert np.array_equal(g, g2) and loss == loss2   # fixed order of sums
    net.close()


def test_training_step_applies_adam_to_the_batch_gradient():
    """One training step on a one-state data set: every row of the batch is
    that state, so the step is Adam's first (m / c1 = g, v / c2 = g^2) on the
    gradient of a batch of one, w - lr g / (|g| + 1e-8)."""
    from cueva.learned import LearnedSeed, synthetic_pairs
    cons, prims = synthetic_pairs(1, seed=9)
    net = LearnedSeed(seed=4)
    net.fit_normalisation(*synthetic_pairs(4096, seed=1))
    g, _ = net.gradients(cons, prims)
    w0 = net.params()[:g.size].astype(np.float64)
    lr = 1e-3
    net.train(cons, prims, steps=1, batch=96, lr=lr, seed=5)
    w1 = net.params()[:g.size].astype(np.float64)
    # 96 equal rows of weight 1/96: the batch gradient equals g to FP32 rounding
    # (96 eps); where |g| >> 1e-8 the step is lr sign(g) to that accuracy, and w
    # itself is rounded to eps |w|
    big = np.abs(g) > 1e-6
    want = -lr * g / (np.abs(g) + 1e-8)
    eps = np.finfo(np.float32).eps
    assert np.all(np.abs((w1 - w0) - want)[big] <= 200 * eps * lr + eps * np.abs(w0[big]))
    net.close()
